"""The clustered FP64 Jacobi solver behind syev / sygv / the reference-mode Rayleigh-Ritz: every cluster size
and the edges between them, odd and even orders, against LAPACK and its own residuals.

Tolerances: a two-sided Jacobi sweep applies at most n - 1 rotations to every row and column, each adding
at most about six roundings (2^-53) of ||A||_F; with at most ten sweeps the backward error is below
60 n 2^-53 ||A||_F, the same bound for the orthogonality of the vectors (||I||_F = sqrt(n) per column is 1)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

U = 2.0 ** -53


@pytest.fixture(scope="module")
def api(built_lib):
    import torch

    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from mixedprecisionofrr_gb300 import api as a

    return a


def _check(A, w, V, M=None):
    n = A.shape[0]
    scale = np.linalg.norm(A) if M is None else np.linalg.norm(A) * np.linalg.norm(np.linalg.inv(M), 2)
    tol = 60 * n * U
    B = V if M is None else M @ V
    cond = 1.0 if M is None else np.linalg.cond(M)
    assert np.all(np.diff(w) >= 0)
    assert np.linalg.norm(A @ V - B * w) <= tol * scale * cond * np.linalg.norm(B, 2)
    assert np.linalg.norm(V.T @ B - np.eye(n), 2) <= tol * cond


def _spectrum(kind, n, rng):
    if kind == "random":
        A = rng.standard_normal((n, n))
        return A + A.T
    Q, _ = np.linalg.qr(rng.standard_normal((n, n)))
    if kind == "graded":
        lam = 10.0 ** (-8.0 * np.arange(n) / max(n - 1, 1))
    else:  # clustered: a few distinct values
        lam = np.repeat([3.0, 1.0, 1.0 - 1e-13, -2.0], -(-n // 4))[:n]
    A = (Q * lam) @ Q.T
    return 0.5 * (A + A.T)


@pytest.mark.parametrize("n", [1, 2, 3, 16, 17, 20, 21, 40, 41, 48, 49, 63, 64, 65, 127, 128, 129, 159, 160, 161])
def test_syev_cluster_edges(api, n):
    rng = np.random.default_rng(n)
    for kind in ("random", "graded", "clustered"):
        A = _spectrum(kind, n, rng)
        w, V = api.syev(A)
        _check(A, w, V)
        assert np.max(np.abs(w - np.linalg.eigvalsh(A))) <= 60 * n * U * np.linalg.norm(A)


@pytest.mark.parametrize("n", [2, 15, 32, 64, 101, 160])
def test_sygv_cluster(api, n):
    rng = np.random.default_rng(100 + n)
    A = _spectrum("random", n, rng)
    X = rng.standard_normal((2 * n + 3, n))
    M = X.T @ X / (2 * n)
    w, V = api.sygv(A, M)
    _check(A, w, V, M)


@pytest.mark.parametrize("b", [1, 7, 16, 32, 64, 80])
def test_zero_diagonal_ties(api, b):
    """[[0, K], [K', 0]]: equal (zero) diagonal entries in every pair of the first round."""
    rng = np.random.default_rng(b)
    K = rng.standard_normal((b, b))
    A = np.block([[np.zeros((b, b)), K], [K.T, np.zeros((b, b))]])
    w, V = api.syev(A)
    _check(A, w, V)
    s = np.linalg.svd(K, compute_uv=False)
    assert np.max(np.abs(w[::-1][:b] - s)) <= 60 * 2 * b * U * np.linalg.norm(A)


def test_scaled_entries(api):
    """Entries far from one (the rotations scale by exponents) and a diagonal input."""
    rng = np.random.default_rng(5)
    A = _spectrum("random", 33, rng)
    w0, _ = api.syev(A)
    for e in (-400, -100, 100, 400):
        w, V = api.syev(np.ldexp(A, e))
        assert np.max(np.abs(np.ldexp(w, -e) - w0)) <= 120 * 33 * U * np.linalg.norm(A)
        assert np.linalg.norm(V.T @ V - np.eye(33), 2) <= 60 * 33 * U
    d = rng.standard_normal(50)
    w, V = api.syev(np.diag(d))
    assert np.array_equal(w, np.sort(d))
