"""MGS without re-orthogonalisation (reorth_tol < 0, or 0, or an orth_tol above every norm) in FP64 keeps the columns that sequential projections keep, also where
columns depend on each other to working precision (Hilbert and Vandermonde blocks); CGS likewise.

Which columns pass select_tol there hangs on rounding: over row permutations the sequential process itself keeps
numbers that differ by at most one, so the GPU's order of sums is allowed two more or fewer than that range."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

EPS = 2.0 ** -52


def _kept(A, stol, classical):
    Q, kept = np.zeros_like(A), []
    for i in range(A.shape[1]):
        v = A[:, i].copy()
        if np.linalg.norm(v) < stol:
            continue
        if classical:
            v = v - Q[:, kept] @ (Q[:, kept].T @ v)
        else:
            for j in kept:
                v = v - (Q[:, j] @ v) * Q[:, j]
        t = np.sqrt(v @ v)
        if t >= stol:
            Q[:, i] = v / t
            kept.append(i)
    return len(kept)


@pytest.mark.parametrize("kind,m,n,stol", [("hilbert", 200, 40, EPS), ("hilbert", 1000, 64, EPS), ("hilbert", 64, 64, EPS),
                                           ("vander", 1000, 64, 1e-14), ("vander", 64, 64, 1e-14),
                                           ("hilbert", 1000, 64, 1e-10)])
@pytest.mark.parametrize("classical,off", [(False, dict(reorth_tol=-1.0)), (False, dict(reorth_tol=0.0)),
                                           (False, dict(orth_tol=1e6)), (True, dict(reorth_tol=-1.0))])
def test_selection_without_reorthogonalisation(built_lib, kind, m, n, stol, classical, off):
    from mixedprecisionofrr_gb300 import api

    if kind == "hilbert":
        A = 1.0 / (np.arange(m)[:, None] + np.arange(n)[None, :] + 1)
    else:
        A = np.vander(np.linspace(0, 1, m), n, increasing=True)
    counts = [_kept(np.ascontiguousarray(A[np.random.default_rng(k).permutation(m)]), stol, classical) for k in range(5)]
    Q, R, skip = api.gs_basis(A, classical, "double", "double", select_tol=stol, **off)
    keep = np.asarray(skip) == 0
    assert min(counts) - 2 <= keep.sum() <= max(counts) + 2
    Q = api.to_numpy(Q)
    # kept columns are reproduced: each projection term adds at most two roundings of the column's norm
    assert np.abs(Q @ R - A)[:, keep].max() <= 4 * n * EPS * np.sqrt(m)
