"""Thick restart of the Krylov eigensolver through the matrix sign function on a cluster (csrc/sign_function.cu): orders
around the row slots (32, 64) and column slots (64) of the kernels, against a dense eigensolver."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kdim", [12, 31, 32, 33, 63, 64, 65, 95])
def test_restarted_eigenvalues(kdim):
    import scipy.sparse as sp

    from mixedprecisionofrr_gb300 import api

    nx = 24
    def one_d(lo, up):
        return sp.diags([np.full(nx - 1, lo), np.full(nx, 2.0), np.full(nx - 1, up)], [-1, 0, 1])
    eye = sp.identity(nx)
    A = (sp.kron(one_d(-1.1, -0.9), eye) + sp.kron(eye, one_d(-1.3, -0.8))).tocsr()  # nonsymmetric, real spectrum
    k = np.arange(1, nx + 1)
    c = np.cos(k * np.pi / (nx + 1))
    lam = (2 - 2 * np.sqrt(0.99) * c)[:, None] + (2 - 2 * np.sqrt(1.04) * c)[None, :]
    nev = 4
    ref = np.sort(lam.ravel())[::-1][:nev]
    v0 = np.random.default_rng(kdim).standard_normal((A.shape[0], 1))
    X, d, info = api.arnoldi_hess_eig(api.CsrMatrix(A), A.shape[0], nev, "double", maxiter=4000, kdim=kdim, v0=v0,
                                      mode="fp64", tol=1e-10)
    d = np.asarray(d.cpu() if hasattr(d, "cpu") else d).ravel()[:nev].real
    # residual tolerance 1e-10 and eigenvalue condition numbers below 1e3 for this grid
    assert np.allclose(np.sort(d)[::-1], ref, rtol=0, atol=1e-6)
