"""FP64 Gram-Schmidt bases built in one cooperative launch, against the oracle's column loop: one CTA and
many, CTAs without rows, rows kept on chip and rows read from memory, the widest on-chip basis and one past
it, dropped columns, a column of NaN, and no re-orthogonalisation.

Tolerance: both are Gram-Schmidt with MGS's (CGS's) error bounds, so a column differs by a modest multiple of
n 2^-53 times the condition number of the columns; 100 n 2^-53 cond is used, on Q (unit columns) and, relative
to the largest entry, on R; Q'Q - I with re-orthogonalisation is below 100 n 2^-53."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

U = 2.0 ** -53


@pytest.fixture(scope="module")
def api(built_lib):
    import torch

    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from mixedprecisionofrr_gb300 import api as a

    return a


@pytest.fixture(scope="module")
def orc():
    from oracle import ofrr_oracle as o

    return o


def _block(m, n, kind, seed):
    rng = np.random.default_rng(seed)
    if kind == "random":
        return rng.standard_normal((m, n))
    r = min(m, n + 16)
    return (rng.standard_normal((m, r)) * 10.0 ** (-3.0 * np.arange(r) / r)) @ rng.standard_normal((r, n))


@pytest.mark.parametrize("classical", [False, True])
@pytest.mark.parametrize("m,n", [(1, 1), (5, 5), (32, 7), (33, 33), (700, 31), (700, 32), (4900, 33), (4864, 1),
                                 (3000, 64), (1500, 127), (1500, 128), (1500, 129), (52000, 40)])
def test_gs_coop_matches_oracle(api, orc, classical, m, n):
    f = orc.cgs if classical else orc.mgs
    for kind in ("random", "correlated") if m < 50000 else ("correlated",):
        A = _block(m, n, kind, m + n)
        Qo, Ro, selo = f(A, "double", "double", full=True)
        Q, R, skip = api.gs_basis(A, classical, "double", "double")
        assert np.array_equal(skip == 0, selo) and not skip.any()
        Qn = api.to_numpy(Q)
        tol = 100 * max(n, 4) * U
        cond = np.linalg.cond(A)
        assert np.max(np.abs(Qn.T @ Qn - np.eye(n))) <= tol
        assert np.max(np.abs(A - Qn @ R)) <= tol * np.max(np.abs(R))
        assert np.max(np.abs(Qn - Qo)) <= tol * cond
        assert np.max(np.abs(R - Ro)) <= tol * cond * np.max(np.abs(Ro))


@pytest.mark.parametrize("classical", [False, True])
@pytest.mark.parametrize("m", [600, 52000])
def test_gs_coop_dropped_and_single_pass(api, orc, classical, m):
    """Zero and dependent columns leave with their flags; reorth_tol < 0 takes one pass per column."""
    f = orc.cgs if classical else orc.mgs
    A = _block(m, 36, "random", 3)
    A[:, 0] = 0.0
    A[:, 9] = A[:, 4] - 2.0 * A[:, 7]
    A[:, 35] = A[:, 34]
    for rt in (None, -1.0):
        Qo, Ro, selo = f(A, "double", "double", select_tol=1e-10, reorth_tol=rt, full=True)
        Q, R, skip = api.gs_basis(A, classical, "double", "double", select_tol=1e-10, reorth_tol=rt)
        assert list(np.flatnonzero(skip)) == [0, 9, 35] and np.array_equal(skip == 0, selo)
        Qn = api.to_numpy(Q)
        tol = 100 * 36 * U * np.linalg.cond(A[:, selo])
        assert np.max(np.abs(Qn - Qo)) <= tol
        assert np.all(Qn[:, skip == 1] == 0.0)
        keep = np.flatnonzero(selo)
        assert np.max(np.abs(R[:, keep] - Ro[:, keep])) <= tol * np.max(np.abs(Ro))


@pytest.mark.parametrize("classical", [False, True])
def test_gs_coop_nan_column(api, classical):
    """A NaN column is kept (no comparison with NaN drops it); the columns before it are untouched."""
    A = _block(900, 12, "random", 8)
    Q0, R0, _ = api.gs_basis(A, classical, "double", "double")
    A[17, 6] = np.nan
    Q, R, skip = api.gs_basis(A, classical, "double", "double")
    assert not skip.any()
    assert np.array_equal(api.to_numpy(Q)[:, :6], api.to_numpy(Q0)[:, :6])
    assert np.array_equal(R[:6, :6], R0[:6, :6])
    assert np.isnan(api.to_numpy(Q)[:, 6:]).all()
