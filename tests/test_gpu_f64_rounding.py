"""Short FP64 reciprocal, quotient and square root (csrc/f64_ops.cuh) where rounding is hardest: quotients, reciprocals and
roots a few units of 2^-107 beside a midpoint between two doubles, and operands a few units in the last place from
values of few bits.  NumPy's own operations are correctly rounded, so the comparison is exact."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _ulps(x, j):
    return (np.asarray(x, np.float64).view(np.int64) + j).view(np.float64)


def _quotients(rng, count):
    """a 2^k = b m + r: a / b = m / 2^k and r / b beside it, m odd of 54 bits, so m / 2^k is a midpoint."""
    a, b = [], []
    while len(a) < count:
        B = int(rng.integers(1 << 52, 1 << 53)) | 1
        for r in (-5, -3, -1, 1, 3, 5):
            for k in (53, 54):
                m = (-r * pow(B, -1, 1 << k)) % (1 << k) | (1 << 53 if k == 53 else 0)
                v = B * m + r
                if m % 2 == 1 and m >> 53 == 1 and v % (1 << k) == 0 and (1 << 52) <= v >> k < (1 << 53):
                    a.append(float(v >> k))
                    b.append(float(B))
    return np.array(a), np.array(b)


def _reciprocals():
    """(2^k + r) / d of 53 bits: the reciprocal is d / 2^k and a small distance, for d of few bits."""
    out = []
    for d in range(3, 600, 2):
        for k in range(52, 64):
            for r in range(-40, 41):
                v = (1 << k) + r
                if v % d == 0:
                    v //= d
                    while v >= 1 << 53 and v % 2 == 0:
                        v //= 2
                    if 1 << 52 <= v < 1 << 53:
                        out.append(float(v))
    return np.array(out)


def _roots(count):
    """m^2 = x 2^s + r with m odd of 54 bits: the root is m / 2 (a midpoint) and a small distance."""
    out = []
    for t in range(-count, count):
        r = 1 + 8 * t
        for s in range(53, 57):
            y = 1
            for k in range(3, s):  # y^2 = r (mod 2^(k + 1))
                if (y * y - r) >> k & 1:
                    y += 1 << (k - 1)
            for m in (y, -y, y + (1 << s - 1), -y + (1 << s - 1)):
                m = m % (1 << s) | (1 << 53 if s == 53 else 0)
                m &= (1 << 54) - 1
                if m >> 53 == 1 and (m * m - r) % (1 << s) == 0:
                    x = (m * m - r) >> s
                    while x >= 1 << 53 and x % 2 == 0:
                        x //= 2
                    if 0 < x < 1 << 53:
                        out.append(float(x << (s & 1)) if x < 1 << 52 else np.ldexp(float(x), s & 1))
    return np.array(out)


def _few_bits():
    c = np.array([1.0, 1.25, 1.5, 1.75, 1.125, 1.375, 1.625, 1.875, 4 / 3, 1.2, 1.6, 8 / 7, 1.0625, 3.0, 5.0, 7.0])
    b = np.concatenate([_ulps(c, j) for j in range(-64, 65)])
    a = np.concatenate([_ulps(c, j) for j in range(-4, 5)])
    return tuple(x.ravel().copy() for x in np.meshgrid(a, b))


def _run(op, a, b, ref):
    import torch

    from mixedprecisionofrr_gb300 import _lib as L
    from mixedprecisionofrr_gb300 import api

    ctx = api.context()
    ad, bd = torch.as_tensor(a, device="cuda"), torch.as_tensor(b, device="cuda")
    out = torch.empty_like(ad)
    torch.cuda.synchronize()
    L.check(ctx.lib.ofrr_debug_f64_ops(ctx.h, op, a.size, ad.data_ptr(), bd.data_ptr(), out.data_ptr()), "f64_ops")
    got = out.cpu().numpy()
    bad = got.view(np.uint64) != ref.view(np.uint64)
    assert not bad.any(), (op, int(bad.sum()), a.size, [float(x).hex() for x in (a[bad][0], b[bad][0], got[bad][0])])


@pytest.mark.parametrize("shift", [0, 37, -300])
def test_beside_midpoints(built_lib, shift):
    rng = np.random.default_rng(11)
    a, b = _quotients(rng, 30000)
    a = np.ldexp(a, shift)
    _run(1, a, b, a / b)
    _run(1, -a, b, -a / b)
    x = np.ldexp(_reciprocals(), shift)
    _run(0, x, x, 1.0 / x)
    x = np.ldexp(_roots(3000), 2 * (shift // 2))
    _run(2, x, x, np.sqrt(x))


def test_beside_values_of_few_bits(built_lib):
    a, b = _few_bits()
    _run(1, a, b, a / b)
    _run(0, b, b, 1.0 / b)
    _run(2, b, b, np.sqrt(b))
