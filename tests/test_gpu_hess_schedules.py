"""Every schedule of the Hessenberg process gives the per-column kernels' basis bit for bit: register panels (16 and 32
columns, part panels, several panels), the blocked cluster form, the cooperative launch and what none of them
holds; heights at the edges of a thread, a warp, a CTA and a cluster, CTAs without rows, ties, a NaN column, a
column of zeros and a dependent one.  The arithmetic is one rounding per operation in a fixed order, so the
comparison is exact."""
import os

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def api(built_lib):
    import torch

    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from mixedprecisionofrr_gb300 import api as a

    return a


def _same(api, A, pc, po, env=None):
    for k, v in (env or {}).items():
        os.environ[k] = v
    try:
        Q, R, sel, perm = api.hessenberg(A, pc, po)
    finally:
        for k in env or {}:
            del os.environ[k]
    os.environ["OFRR_HESS_PER_COLUMN"] = "1"
    try:
        Qc, Rc, selc, permc = api.hessenberg(A, pc, po)
    finally:
        del os.environ["OFRR_HESS_PER_COLUMN"]
    assert np.array_equal(sel, selc) and np.array_equal(perm, permc)
    assert np.array_equal(R, Rc, equal_nan=True)
    assert np.array_equal(api.to_numpy(Q), api.to_numpy(Qc), equal_nan=True)


def _block(m, n, seed, dt):
    rng = np.random.default_rng(seed)
    r = min(m, n + 8)
    A = (rng.standard_normal((m, r)) * 10.0 ** (-2.0 * np.arange(r) / r)) @ rng.standard_normal((r, n))
    return (A / np.abs(A).max(0)).astype(dt)


@pytest.mark.parametrize("pc,po", [("single", "half"), ("single", "single"), ("double", "double"), ("double", "half"),
                                   ("single", "double")])
@pytest.mark.parametrize("m,n", [(16, 16), (17, 3), (33, 33), (511, 16), (513, 17), (2048, 32), (4097, 48), (8192, 33),
                                 (8192, 64), (8193, 20), (9000, 65), (300, 100), (20000, 40)])
def test_schedules_bit_identical(api, orc_dt, m, n, pc, po):
    _same(api, _block(m, n, m + n, orc_dt(po)), pc, po)


@pytest.fixture(scope="module")
def orc_dt():
    from oracle import ofrr_oracle as o

    return o._dt


@pytest.mark.parametrize("pc,po", [("single", "half"), ("double", "double")])
@pytest.mark.parametrize("m", [600, 8192, 26000, 110000])
def test_schedules_special_columns(api, orc_dt, m, pc, po):
    """Ties in a column (equal maxima in several CTAs), a zero column, a repeated column and a NaN column."""
    A = _block(m, 40, 9, orc_dt(po))
    A[:, 5] = 0
    A[[3, m // 2, m - 1], 0] = 1
    A[:, 21] = A[:, 20]
    _same(api, A, pc, po)
    A[:, 30] = np.nan
    _same(api, A, pc, po)


@pytest.mark.parametrize("m,n", [(3000, 40), (4096, 33), (8192, 40)])
def test_portable_cluster(api, orc_dt, m, n):
    _same(api, _block(m, n, 2, orc_dt("half")), "single", "half", {"OFRR_HESS_CLUSTER": "8"})
