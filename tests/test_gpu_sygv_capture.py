"""ofrr_syev / ofrr_sygv queue work on the context's stream and read nothing from the host afterwards, so a caller may
capture them in a CUDA graph and run it again on new matrices in the same buffers.

Tolerance: as in the solvers' own tests, 60 n 2^-53 ||A||_F for the eigenvalues, times ||M^-1||_2 and cond(M) for the
pencil."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

U = 2.0 ** -53


@pytest.mark.parametrize("pencil", [False, True])
@pytest.mark.parametrize("n", [5, 32, 64, 101, 144])
def test_captured_solver_follows_its_inputs(built_lib, n, pencil):
    import scipy.linalg as sl
    import torch

    from mixedprecisionofrr_gb300 import _lib as L
    from mixedprecisionofrr_gb300 import api

    ctx = api.context()
    rng = np.random.default_rng(n)

    def problem():
        A, B = rng.standard_normal((n, n)), rng.standard_normal((n, n))
        return A + A.T, B @ B.T / n + np.eye(n)

    def load(A, M):
        Ad.copy_(torch.as_tensor(A).cuda())
        Md.copy_(torch.as_tensor(M).cuda())

    def solve():
        if pencil:
            return ctx.lib.ofrr_sygv(ctx.h, n, Ad.data_ptr(), n, Md.data_ptr(), n, w.data_ptr())
        return ctx.lib.ofrr_syev(ctx.h, n, Ad.data_ptr(), n, w.data_ptr())

    Ad, Md, w = api.empty_cm(n, n, L.F64), api.empty_cm(n, n, L.F64), torch.zeros(n, dtype=torch.float64, device="cuda")
    load(*problem())
    L.check(solve(), "first call")  # the workspace and the library's module are there before the capture
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g, stream=torch.cuda.current_stream()):
        status = solve()
    L.check(status, "captured call")
    api.sygv(*problem())  # other work through the same context and host stack
    for _ in range(2):
        A, M = problem()
        load(A, M)
        g.replay()
        torch.cuda.synchronize()
        M = M if pencil else np.eye(n)
        ref = sl.eigh(A, M, eigvals_only=True)
        tol = 60 * n * U * np.linalg.norm(A) * np.linalg.norm(np.linalg.inv(M), 2) * np.linalg.cond(M)
        assert np.max(np.abs(w.cpu().numpy() - ref)) <= tol
        V = Ad.cpu().numpy()
        assert np.linalg.norm(A @ V - (M @ V) * ref) <= tol * np.linalg.norm(M @ V, 2)
