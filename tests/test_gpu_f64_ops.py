"""Short FP64 reciprocal, quotient and square root (csrc/f64_ops.cuh): correctly rounded on random significands over the
whole exponent range (short path, its limits, and the operands that take the plain operation), on significands at the
ends of their range, and on special values."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _operands(kind, n, rng):
    frac = rng.integers(0, 2**52, n, dtype=np.uint64)
    if kind == "edges":  # significands next to 1 and 2, and with few bits
        frac = np.where(rng.random(n) < 0.5, frac >> rng.integers(20, 53, n).astype(np.uint64),
                        np.uint64(2**52 - 1) - (frac >> rng.integers(20, 53, n).astype(np.uint64)))
    lo, hi = {"near": (1000, 1046), "wide": (1, 2046), "limits": (190, 210), "top": (1840, 1850), "edges": (900, 1150)}[kind]
    e = rng.integers(lo, hi + 1, n).astype(np.uint64)
    s = rng.integers(0, 2, n).astype(np.uint64)
    return (frac | (e << np.uint64(52)) | (s << np.uint64(63))).view(np.float64)


@pytest.mark.parametrize("kind", ["near", "wide", "limits", "top", "edges", "special"])
def test_correctly_rounded(kind):
    import torch

    from mixedprecisionofrr_gb300 import _lib as L
    from mixedprecisionofrr_gb300 import api

    rng = np.random.default_rng(5)
    if kind == "special":
        v = np.array([0.0, -0.0, 1.0, -1.0, 2.0, 4.0, 0.5, np.inf, -np.inf, np.nan, 5e-324, 2.2e-308, 1.7e308, 3.0])
        a, b = (x.ravel().copy() for x in np.meshgrid(v, v))
    else:
        a, b = _operands(kind, 1 << 20, rng), _operands(kind, 1 << 20, rng)
    ctx = api.context()
    Ad, Bd = torch.as_tensor(a, device="cuda"), torch.as_tensor(b, device="cuda")
    out = torch.empty_like(Ad)
    with np.errstate(all="ignore"):
        refs = [1.0 / a, a / b, np.sqrt(np.abs(a))]
    for op, ref in enumerate(refs):
        x = Ad.abs() if op == 2 else Ad
        torch.cuda.synchronize()
        L.check(ctx.lib.ofrr_debug_f64_ops(ctx.h, op, a.size, x.data_ptr(), Bd.data_ptr(), out.data_ptr()), "f64_ops")
        got = out.cpu().numpy()
        same = (got.view(np.uint64) == ref.view(np.uint64)) | (np.isnan(got) & np.isnan(ref))
        assert np.all(same), (op, a[~same][:3], b[~same][:3], got[~same][:3], ref[~same][:3], int((~same).sum()))
