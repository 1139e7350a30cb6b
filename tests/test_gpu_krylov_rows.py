"""Krylov steps on rows of different lengths (csrc/krylov_tr.cu: kry_extend takes pivot rows of up to 8 nonzeros eight lanes
at a time and longer ones a warp at a time): leading eigenvalues of a diagonally scaled symmetric matrix."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mode,prec", [("fp64", "double"), ("mixed", "single")])
@pytest.mark.parametrize("width", [1, 7, 8, 9, 40])
def test_row_lengths(width, mode, prec):
    import scipy.sparse as sp

    from mixedprecisionofrr_gb300 import api

    n, nev = 500, 4
    rng = np.random.default_rng(width)
    rows = np.repeat(np.arange(n), width)
    cols = (rows + rng.integers(0, n, rows.size)) % n
    off = sp.coo_matrix((rng.standard_normal(rows.size) * 0.02, (rows, cols)), shape=(n, n))
    S = sp.csr_matrix(off + off.T + sp.diags(np.linspace(1.0, 2.0, n) ** 6))
    ref = np.linalg.eigvalsh(S.toarray())[::-1][:nev]
    t = np.exp(rng.uniform(-0.5, 0.5, n))
    A = (sp.diags(1.0 / t) @ S @ sp.diags(t)).tocsr()  # the same eigenvalues, not symmetric
    X, d, info = api.arnoldi_hess_eig(api.CsrMatrix(A), n, nev, prec, "half" if mode == "mixed" else None, maxiter=6000,
                                      kdim=30, v0=rng.standard_normal((n, 1)), mode=mode, tol=1e-9)
    assert info.status == 0, info
    # relative residual 1e-9, eigenvalue condition numbers at most cond(diag(t)) = e
    assert np.max(np.abs(np.sort(np.asarray(d))[::-1][:nev] - ref)) <= 1e-8 * ref[0]
