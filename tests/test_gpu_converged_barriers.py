"""Kernels whose warps reach a cluster's or a named barrier from uneven loops and one-sided stores (clustered Jacobi
sweeps, sign function, nonsymmetric QR with its second warp): repeated beside another stream's kernels, which delay
single warps, they end and give the same bits every time, at orders that leave warps and lanes without work."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _load(torch, side, a):
    with torch.cuda.stream(side):
        for _ in range(6):
            a.mul_(1.0000001)


@pytest.mark.parametrize("n", [22, 41, 57, 99, 143])
def test_jacobi_repeats(built_lib, n):
    import torch

    from mixedprecisionofrr_gb300 import api

    api.context()
    rng = np.random.default_rng(n)
    A = rng.standard_normal((n, n))
    A = A + A.T
    side, a = torch.cuda.Stream(), torch.ones(1 << 22, device="cuda")
    torch.cuda.synchronize()
    w0, V0 = api.syev(A)
    for _ in range(15):
        _load(torch, side, a)
        w, V = api.syev(A)
        assert np.array_equal(w, w0) and np.array_equal(V, V0)
    torch.cuda.synchronize()


@pytest.mark.parametrize("kdim", [21, 34, 66])
def test_krylov_restart_repeats(built_lib, kdim):
    import scipy.sparse as sp
    import torch

    from mixedprecisionofrr_gb300 import api

    nx = 20
    d1 = sp.diags([np.full(nx - 1, -1.2), np.full(nx, 2.0), np.full(nx - 1, -0.8)], [-1, 0, 1])
    A = (sp.kron(d1, sp.identity(nx)) + sp.kron(sp.identity(nx), d1)).tocsr()
    C = api.CsrMatrix(A)
    v0 = np.random.default_rng(kdim).standard_normal((A.shape[0], 1))
    side, a = torch.cuda.Stream(), torch.ones(1 << 22, device="cuda")
    torch.cuda.synchronize()
    runs = []
    for _ in range(4):
        _load(torch, side, a)
        X, d, _ = api.arnoldi_hess_eig(C, A.shape[0], 4, "double", maxiter=300, kdim=kdim, v0=v0, mode="fp64", tol=1e-10)
        runs.append((api.to_numpy(X), np.asarray(d.cpu() if hasattr(d, "cpu") else d)))
    for X, d in runs[1:]:
        assert np.array_equal(X, runs[0][0], equal_nan=True) and np.array_equal(d, runs[0][1], equal_nan=True)
    torch.cuda.synchronize()
