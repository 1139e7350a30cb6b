"""CSR products over the forms a launch distinguishes: one, up to four and more right-hand sides with a partial
last chunk, row blocks with a remainder, rows whose nonzeros fit the CTA's staging and rows that do not, empty
rows and columns, duplicate entries; and the transpose behind 'T' at the edges of its scan.

Tolerance: an output entry is a sum of k products in the compute type; every product and sum rounds once at
most, so its error is below (k + 1) u |A||X| with the compute type's u (plus one rounding of X and of the
values, already exact here for FP64, 2^-24 each for FP32)."""
import numpy as np
import pytest
import scipy.sparse as sp

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def api(built_lib):
    import torch

    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from mixedprecisionofrr_gb300 import api as a

    return a


def _random_csr(m, n, per_row, seed, dense_rows=0):
    rng = np.random.default_rng(seed)
    lens = rng.integers(0, per_row + 1, m)
    if dense_rows:
        lens[rng.choice(m, dense_rows, replace=False)] = n
    ptr = np.concatenate([[0], np.cumsum(lens)]).astype(np.int32)
    idx = np.concatenate([np.sort(rng.choice(n, l, replace=False)) for l in lens] + [np.zeros(0, int)]).astype(np.int32)
    return {"indptr": ptr, "indices": idx, "a_double": rng.standard_normal(len(idx)), "nrows": m, "ncols": n}


def _check(api, A, trans, nrhs, pc, pin, seed):
    S = sp.csr_matrix((A["a_double"], A["indices"], A["indptr"]), shape=(A["nrows"], A["ncols"]))
    S = S.T.tocsr() if trans == "T" else S
    X = np.random.default_rng(seed).standard_normal((S.shape[1], nrhs))
    X = X.astype({"double": np.float64, "single": np.float32, "half": np.float16}[pin])
    from mixedprecisionofrr_gb300 import _lib as L

    Xd = api.to_device_cm(X, {"double": L.F64, "single": L.F32, "half": L.F16}[pin])
    Y = api.to_numpy(api.csrmv(api.CsrMatrix(A, symmetric=False), trans, Xd, pc)).astype(np.float64)
    k = int(np.diff(S.indptr).max(initial=0))
    u = 2.0 ** -53 if pc == "double" else 2.0 ** -24
    bound = (k + 4) * u * (abs(S) @ np.abs(X.astype(np.float64))) + 1e-300
    assert np.all(np.abs(Y - S @ X.astype(np.float64)) <= bound)


@pytest.mark.parametrize("trans", ["N", "T"])
@pytest.mark.parametrize("pc,pin", [("double", "double"), ("single", "single"), ("single", "half"), ("double", "single")])
def test_right_hand_side_chunks(api, trans, pc, pin):
    A = _random_csr(515, 301, 9, 1)
    for nrhs in (1, 2, 3, 4, 5, 8, 9, 16, 23, 65):
        _check(api, A, trans, nrhs, pc, pin, nrhs)


@pytest.mark.parametrize("trans", ["N", "T"])
@pytest.mark.parametrize("m,n,per_row,dense", [(1, 1, 1, 0), (255, 40, 5, 0), (256, 4095, 5, 0), (257, 4096, 7, 0),
                                               (4097, 4097, 3, 0), (600, 900, 12, 3), (40, 9000, 4, 1), (3, 5, 0, 0)])
def test_row_blocks_and_scan_edges(api, trans, m, n, per_row, dense):
    A = _random_csr(m, n, per_row, m + n, dense)
    if len(A["indices"]) == 0:  # an operator without values is refused, as before
        with pytest.raises(Exception, match="1000"):
            _check(api, A, trans, 3, "double", "double", 7)
        return
    _check(api, A, trans, 3, "double", "double", 7)
    _check(api, A, trans, 17, "single", "single", 8)


def test_transpose_with_duplicates_is_deterministic(api):
    """Entries given twice keep the input's order in the transpose: 'T' equals 'N' of the transpose built on the
    host, bit for bit, and runs agree."""
    rng = np.random.default_rng(4)
    m, n, k = 700, 50, 6
    ptr = (np.arange(m + 1) * k).astype(np.int32)
    idx = rng.integers(0, n, m * k).astype(np.int32)  # unsorted, with repeats
    val = rng.standard_normal(m * k)
    rows = np.repeat(np.arange(m), k)
    o = np.lexsort((np.arange(m * k), rows, idx))
    tp = np.concatenate([[0], np.cumsum(np.bincount(idx, minlength=n))]).astype(np.int32)
    X = rng.standard_normal((m, 5))
    A = api.CsrMatrix({"indptr": ptr, "indices": idx, "a_double": val, "nrows": m, "ncols": n}, symmetric=False)
    T = api.CsrMatrix({"indptr": tp, "indices": rows[o].astype(np.int32), "a_double": val[o], "nrows": n, "ncols": m},
                      symmetric=False)
    Y = [api.to_numpy(api.csrmv(A, "T", X, "double")) for _ in range(3)]
    assert np.array_equal(Y[0], Y[1]) and np.array_equal(Y[0], Y[2])
    assert np.array_equal(Y[0], api.to_numpy(api.csrmv(T, "N", X, "double")))
