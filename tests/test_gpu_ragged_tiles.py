"""16-bit and exact-slice products whose last tiles are ragged (lanes of a warp with and without rows or columns to store,
between the aligned transfers of the next columns): right against FP64, and the same bits beside another stream's
kernels.  FP32 sums of exact products: K 2^-24 of |A|'|B|; the exact-slice product's documented 2^-33."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("M,N,K", [(1, 65, 64), (129, 96, 200), (255, 127, 640), (4001, 33, 300), (77, 128, 2048)])
def test_ragged(built_lib, M, N, K):
    import torch

    from mixedprecisionofrr_gb300 import api

    api.context()
    g = torch.Generator(device="cuda").manual_seed(M + N + K)
    A = torch.randn(K, M, generator=g, device="cuda", dtype=torch.float64)
    B = torch.randn(K, N, generator=g, device="cuda", dtype=torch.float64)
    Ah, Bh = A.half().t().contiguous().t(), B.half().t().contiguous().t()
    side, a = torch.cuda.Stream(), torch.ones(1 << 22, device="cuda")
    ref, bound = A.t() @ B, A.abs().t() @ B.abs()
    refh = Ah.double().t() @ Bh.double()
    torch.cuda.synchronize()
    C0, E0 = api.gemm(Ah, "T", Bh, "single", "single"), api.gemm_f64_emulated(A, B)
    assert bool(((C0.double() - refh).abs() <= 1.01 * K * 2.0 ** -24 * (Ah.double().abs().t() @ Bh.double().abs())).all())
    assert bool(((E0 - ref).abs() <= 2.0 ** -33 * bound).all())
    for _ in range(10):
        with torch.cuda.stream(side):
            a.mul_(1.0000001)
        assert torch.equal(api.gemm(Ah, "T", Bh, "single", "single"), C0)
        assert torch.equal(api.gemm_f64_emulated(A, B), E0)
    torch.cuda.synchronize()
