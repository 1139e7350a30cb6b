"""Transposed CSR products of a matrix with one dense column (a constraint column, an arrow matrix): the column's nonzeros are
ranked against each other, and the transposed row is one thread's chain.  Also with entries of that column repeated."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("pc", ["double", "single"])
@pytest.mark.parametrize("length", [31, 1024, 20000])
def test_dense_column(built_lib, length, pc):
    import scipy.sparse as sp
    import torch

    from mixedprecisionofrr_gb300 import api

    api.context()
    rng = np.random.default_rng(length)
    m, n = 25000, 3000
    heavy = np.sort(rng.choice(m, length, replace=False))
    rows = np.concatenate([np.arange(m), heavy, heavy[:5]])
    cols = np.concatenate([rng.integers(0, n, m), np.full(length, 7), np.full(5, 7)])  # five entries twice
    vals = rng.standard_normal(rows.size)
    order = np.argsort(rows, kind="stable")
    rows, cols, vals = rows[order], cols[order], vals[order]
    ptr = np.searchsorted(rows, np.arange(m + 1)).astype(np.int32)
    C = api.CsrMatrix.from_device(torch.as_tensor(ptr).cuda(), torch.as_tensor(cols.astype(np.int32)).cuda(),
                                  torch.as_tensor(vals).cuda(), (m, n))
    dt = np.float64 if pc == "double" else np.float32
    X = rng.standard_normal((m, 3)).astype(dt)
    Y = api.to_numpy(api.csrmv(C, "T", X, pc))
    A = sp.csr_matrix((vals.astype(dt).astype(np.float64), cols, ptr), shape=(m, n))
    ref = A.T @ X.astype(np.float64)
    bound = abs(A).T @ np.abs(X.astype(np.float64))
    # one chain of FMAs: at most `nonzeros of the column` roundings of sums below the bound
    k = np.bincount(cols, minlength=n)[:, None]
    assert np.all(np.abs(Y - ref) <= 1.01 * (k + 1) * np.finfo(dt).eps * bound)
    again = api.to_numpy(api.csrmv(C, "T", X, pc))
    assert np.array_equal(Y, again)  # whatever order the nonzeros arrived in
