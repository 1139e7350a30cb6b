"""A wait that runs out in a warp-wide loop: lanes with different limits, one of them past its wait at once, leave the
loop together, the launch ends, the status is reported once, and the kernels that wait this way (16-bit product,
exact-slice product, batched eigensolver) still give their results."""
import time

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("timeout_ms", [1, 30])
def test_lanes_leave_together(built_lib, timeout_ms):
    import torch

    from mixedprecisionofrr_gb300 import _lib as L
    from mixedprecisionofrr_gb300 import api

    ctx = api.context()
    assert ctx.lib.ofrr_ctx_synchronize(ctx.h) == L.SUCCESS
    t0 = time.time()
    assert ctx.lib.ofrr_debug_bounded_wait(ctx.h, timeout_ms * 1_000_000) == L.SUCCESS
    assert ctx.lib.ofrr_ctx_synchronize(ctx.h) == 6004  # OFRR_ERR_DEVICE_TIMEOUT
    assert timeout_ms / 1000.0 <= time.time() - t0 < 1.0
    assert ctx.lib.ofrr_ctx_synchronize(ctx.h) == L.SUCCESS

    rng = np.random.default_rng(timeout_ms)
    A, B = rng.standard_normal((500, 300)), rng.standard_normal((500, 24))
    bound = np.abs(A).T @ np.abs(B)
    got = api.gemm_f64_emulated(A, B).cpu().numpy()
    assert np.all(np.abs(got - A.T @ B) <= 2.0 ** -33 * bound)
    h = api.gemm(torch.as_tensor(A).half().cuda(), "T", torch.as_tensor(B).half().cuda(), "single", "single").cpu().numpy()
    ref = A.astype(np.float16).astype(np.float64).T @ B.astype(np.float16).astype(np.float64)
    assert np.all(np.abs(h - ref) <= 500 * 2.0 ** -24 * 1.01 * bound)  # FP32 sums of exact products

    n = 200
    lam = np.linspace(1.0, 0.01, n)
    Q, _ = np.linalg.qr(rng.standard_normal((n, n)))
    S = (Q * lam) @ Q.T
    buf = torch.as_tensor(0.5 * (S + S.T)).reshape(-1).cuda()
    _, ev, _, _, st = api.batch_sym_eig(buf, np.array([n], np.int64), np.array([0], np.int64), nev=4, tol=1e-8)
    # a unit vector of residual r <= 1e-8 (relative to the norm 1) has its Rayleigh quotient within r of an eigenvalue
    assert np.all(np.asarray(st) == 0) and np.abs(np.asarray(ev)[0, :4] - lam[:4]).max() <= 1e-8
