"""FP64 Rayleigh-Ritz step on a symmetric operator (csrc/gram_pair.cu): block widths at the edges of the 4 x 4 blocks, of
the row slices and of one CTA's share, and row counts below and above one slab and one chunk per SM."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("b", [1, 3, 4, 5, 16, 33, 64, 65, 76, 77, 127, 128])
@pytest.mark.parametrize("n", [130, 700, 5000, 12001])
def test_eig_rr_widths(n, b):
    import scipy.linalg as sl
    import scipy.sparse as sp

    from mixedprecisionofrr_gb300 import api

    A = sp.diags([np.full(n - 1, -1.0), np.linspace(2.0, 5.0, n), np.full(n - 1, -1.0)], [-1, 0, 1]).tocsr()
    V = np.random.default_rng(1000 * b + n).standard_normal((n, b))
    X, d = api.eig_rr(api.CsrMatrix(A), V, "double", use_generalized=True, symmetric=True)
    X, d = api.to_numpy(X), np.asarray(d.cpu() if hasattr(d, "cpu") else d).ravel()
    w = sl.eigh(V.T @ (A @ V), V.T @ V, eigvals_only=True)[::-1]
    # eigenvalue error of the pencil: a few n eps ||A|| cond(V'V); cond is below 1e4 for these shapes (n = 130, b = 128:
    # a nearly square Gaussian, below 1e7)
    cond = np.linalg.cond(V) ** 2
    assert np.max(np.abs(d - w)) <= 50 * n * 2.2e-16 * 7.0 * max(cond, 10.0) + 1e-9 * 7.0
    R = V.T @ (A @ X - X * d[None, :])  # Galerkin condition
    assert np.max(np.abs(R)) <= 1e-9 * np.linalg.norm(V) * np.linalg.norm(X) * max(cond, 10.0) ** 0.5
