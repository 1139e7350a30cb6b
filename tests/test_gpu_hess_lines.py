"""Hessenberg bases on both sides of the lines between the schedules (columns and rows at which a one-launch basis takes
over from the blocked ones): bit for bit the per-column kernels' basis, as everywhere."""
import os

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("pc,po,m,n", [("single", "half", m, n) for m in (32768, 32769) for n in (80, 81)]
                         + [("single", "single", 32769, 17), ("single", "bfloat16", 33000, 16)]
                         + [("double", "double", m, n) for m, n in ((4096, 32), (4096, 33), (4097, 32), (4097, 16),
                                                                    (8192, 16), (8192, 17), (8193, 16), (8193, 1))])
def test_lines(built_lib, pc, po, m, n):
    import torch

    from mixedprecisionofrr_gb300 import api

    api.context()
    dt = {"half": torch.float16, "bfloat16": torch.bfloat16, "single": torch.float32, "double": torch.float64}[po]
    g = torch.Generator(device="cuda").manual_seed(m * n)
    X = torch.randn(m, n + 4, generator=g, device="cuda", dtype=torch.float64)
    X = X @ torch.randn(n + 4, n, generator=g, device="cuda", dtype=torch.float64)
    X = (X / X.abs().amax(0)).to(dt)
    Q, R, sel, perm = api.hessenberg(X, pc, po)
    os.environ["OFRR_HESS_PER_COLUMN"] = "1"
    try:
        Qc, Rc, selc, permc = api.hessenberg(X, pc, po)
    finally:
        del os.environ["OFRR_HESS_PER_COLUMN"]
    assert torch.equal(Q, Qc) and np.array_equal(R, Rc)
    assert np.array_equal(sel, selc) and np.array_equal(perm, permc)
