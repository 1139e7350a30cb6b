"""K ranges of the 16-bit tensor-core product summed inside a thread-block cluster (csrc/gemm_tc.cu: cluster_reduce).

Small integer operands: every partial sum is exact in FP32 and every result is exact in the output type, so the product
is compared for equality at ragged rows, columns and K, for each tile width (N) and each cluster size.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("splits", [2, 4, 8])
@pytest.mark.parametrize("M,N,K", [(1, 1, 512), (127, 31, 520), (128, 32, 1024), (129, 33, 577), (200, 64, 1000),
                                   (300, 100, 2047), (77, 129, 513)])
@pytest.mark.parametrize("out", ["single", "half"])
def test_cluster_sum_exact(monkeypatch, splits, M, N, K, out):
    from mixedprecisionofrr_gb300 import api

    rng = np.random.default_rng(M * 7 + N * 3 + K)
    A = rng.integers(-2, 3, size=(K, M)).astype(np.float64)
    B = rng.integers(-2, 3, size=(K, N)).astype(np.float64)
    ref = A.T @ B
    assert np.abs(ref).max() <= 2048  # exact in FP16
    monkeypatch.setenv("OFRR_TC_SPLITS", str(splits))
    Ad, Bd = (api.to_device_cm(X, api.PREC["half"]) for X in (A, B))
    assert np.array_equal(api.gemm(Ad, "T", Bd, "single", out).double().cpu().numpy(), ref)
