"""Row tiles of the batched eigensolver's products (csrc/batch_eig.cu: be_layout picks thread groups and rows per thread
from n): matrices at the edges of every layout, with and without rows past the padded leading dimension."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("sizes", [[16, 31, 32, 33, 63, 65, 95, 97], [127, 128, 129, 159, 161, 191, 193, 255, 257],
                                   [319, 321, 383, 385, 511, 513, 639, 641], [767, 769, 1023, 1024]])
@pytest.mark.parametrize("p16", ["bfloat16", "half"])
def test_layout_edges(sizes, p16):
    import torch

    from mixedprecisionofrr_gb300 import api

    rng = np.random.default_rng(sizes[0])
    mats, lams = [], []
    for n in sizes:
        lam = np.concatenate([np.linspace(10.0, 6.0, 8), rng.uniform(0.0, 3.0, n - 8)])  # the wanted pairs well apart
        Q, _ = np.linalg.qr(rng.standard_normal((n, n)))
        A = (Q * lam) @ Q.T
        mats.append(0.5 * (A + A.T))
        lams.append(lam[:8])
    ns = np.array(sizes, dtype=np.int64)
    offs = np.concatenate([[0], np.cumsum(ns * ns)[:-1]]).astype(np.int64)
    Ad = torch.as_tensor(np.concatenate([m.ravel() for m in mats]), device="cuda")
    Xs, ev, res, its, sts = api.batch_sym_eig(Ad, ns, offs, nev=8, tol=1e-7, p_output=p16)
    assert np.all(sts == 0), (sts, res.max(axis=1))
    for i, A in enumerate(mats):
        X = api.to_numpy(Xs[i])
        r = np.linalg.norm(A @ X - X * ev[i][None, :], axis=0) / (10.0 * np.linalg.norm(X, axis=0))
        assert np.max(r) <= 1.01e-7, (sizes[i], r)
        # a symmetric matrix's eigenvalue error is at most the residual norm
        assert np.max(np.abs(ev[i] - lams[i])) <= 1.01e-6, (sizes[i], ev[i] - lams[i])
