"""Packed digits of the left operand of the exact-slice FP64 product (csrc/sliced.cu: slice_pack, k_sliced_tn).

Against unit columns every digit pair that carries information is kept, so C = A' B returns the left operand rounded to
35 bits below its column's power of two, with no other error: each digit's packing and unpacking, the rows and columns
beyond the last tile and the zero padding of K are compared exactly.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("K", [1, 2, 63, 64, 65, 200, 600, 1025, 4097, 8193])
@pytest.mark.parametrize("M", [1, 127, 129])
def test_unit_columns_return_the_digits(K, M):
    from mixedprecisionofrr_gb300 import api

    rng = np.random.default_rng(K * 1000 + M)
    N = min(K, 65)
    A = rng.integers(-(2**35) + 1, 2**35, size=(K, M)).astype(np.float64)
    special = np.array([2.0**35 - 1, -(2.0**35) + 1, 2.0**35 - 0.5, -(2.0**35) + 0.5, 0.0, 1.0, -1.0, 64.0, -64.0, 63.0])
    A[rng.integers(0, K, 4 * M), np.repeat(np.arange(M), 4)] = rng.choice(special, 4 * M)
    A[K - 1, :] = np.where(rng.random(M) < 0.5, 2.0**34, -(2.0**35) + 1)  # the column's exponent: 35
    rows = rng.permutation(K)[:N]
    B = np.zeros((K, N))
    B[rows, np.arange(N)] = 1.0
    C = api.gemm_f64_emulated(A, B).cpu().numpy()
    assert np.array_equal(C, np.rint(A[rows, :]).T)
