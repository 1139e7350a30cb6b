"""The register panels' exchange under load: many builds of one basis beside another stream's kernels, which delay single
warps and CTAs, all give the per-column kernels' basis.  (Every warp of a CTA decides from the same reduction entries
which of them sends the CTA's candidate, so entries that change while a delayed warp reads them give other bits, or a
bounded wait that runs out.)"""
import os

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("po", ["half", "bfloat16", "single"])
@pytest.mark.parametrize("m,n", [(8192, 64), (8191, 33), (2048, 16)])
def test_panels_under_load(built_lib, m, n, po):
    import torch

    from mixedprecisionofrr_gb300 import api

    api.context()
    g = torch.Generator(device="cuda").manual_seed(m + n)
    dt = {"half": torch.float16, "bfloat16": torch.bfloat16, "single": torch.float32}[po]
    X = torch.randn(m, n + 8, generator=g, device="cuda") @ torch.randn(n + 8, n, generator=g, device="cuda")
    X = (X / X.abs().amax(0)).to(dt).t().contiguous().t()
    os.environ["OFRR_HESS_PER_COLUMN"] = "1"
    try:
        Q0, R0, sel0, perm0 = api.hessenberg(X, "single", po)
    finally:
        del os.environ["OFRR_HESS_PER_COLUMN"]
    side = torch.cuda.Stream()
    a = torch.randn(1 << 22, device="cuda")
    b = torch.randn(512, 512, device="cuda")
    torch.cuda.synchronize()
    for _ in range(40):
        with torch.cuda.stream(side):
            for _ in range(4):
                a.mul_(1.0000001)
                b = torch.tanh(b @ b)
        Q, R, sel, perm = api.hessenberg(X, "single", po)
        assert torch.equal(Q, Q0) and np.array_equal(R, R0)
        assert np.array_equal(sel, sel0) and np.array_equal(perm, perm0)
    torch.cuda.synchronize()
