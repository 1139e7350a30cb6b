"""FP32 arithmetic with FP64 storage, odd widths: the per-column Hessenberg kernels keep the pivot rows' values in
shared memory behind n FP32 coefficients, and those values are eight bytes wide.  Bit-identical to the oracle
(one rounding per operation)."""
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


@pytest.fixture(scope="module")
def orc():
    from oracle import ofrr_oracle as o

    return o


@pytest.mark.parametrize("m,n", [(17, 3), (300, 7), (1000, 21), (300, 8)])
@pytest.mark.parametrize("per_column", [False, True])
def test_single_compute_double_storage(api, orc, m, n, per_column):
    A = np.random.default_rng(m + n).uniform(-1, 1, (m, n))
    if per_column:
        os.environ["OFRR_HESS_PER_COLUMN"] = "1"
    try:
        Q, R, sel, perm = api.hessenberg(A, "single", "double")
    finally:
        os.environ.pop("OFRR_HESS_PER_COLUMN", None)
    Qo, Ro, selo, permo = orc.hessenberg(A, "single", "double")
    assert np.array_equal(sel, selo) and np.array_equal(perm, permo)
    assert np.array_equal(api.to_numpy(Q), Qo)
