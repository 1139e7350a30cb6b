"""The work that is timed: single calls of the solvers' building blocks and whole solves, each through the
package's public functions, at the sizes of the repository's own workloads (the 8192 x 2048 truncated SVD, the
3-D convection-diffusion operator, the batch of dense symmetric matrices, the 2-D/3-D Dirichlet Laplacians) and
over the ranges of its serving stream and tests.

A case is a dict with a "kind" and sizes; `listed()` gives the fixed ones, `draw(rng)` one more of the same
ranges.  Inputs are made on the GPU from the seed alone; `exact` restates a call in 64 bits with plain torch.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from mixedprecisionofrr_gb300 import api

F64 = torch.float64
TORCH = {"double": torch.float64, "single": torch.float32, "half": torch.float16, "bfloat16": torch.bfloat16}
BYTES = {"double": 8, "single": 4, "half": 2, "bfloat16": 2}


# ---- the cases ------------------------------------------------------------------------------------------
def listed():
    return [
        # a small symmetric eigenproblem through the MATLAB-mirror call with its default arithmetic (FP64): the
        # 64-wide 2-D Laplacian, 16 columns; launches and the small projected pencil count here
        {"name": "si_eig_lap_64x65_k16", "kind": "si_eig", "nx": 64, "ny": 65, "nz": 1, "k": 16, "maxiter": 8, "step": 2},
        # the truncated SVD the benchmark reports: top 32 triplets to 1e-8, 16-bit phase, then FP64 accuracy
        {"name": "svd_mixed_8192x2048", "kind": "svd_mixed", "m": 8192, "n": 2048, "block": 64, "nev": 32, "step": 8,
         "step64": 12, "tol": 1e-8, "factors": "dense"},
        # the nonsymmetric sparse Krylov solve (thick-restart Hessenberg process, kdim 64) on a 64^3 grid
        {"name": "krylov_mixed_64c", "kind": "krylov", "n1": 64, "nev": 20, "kdim": 64, "mode": "mixed", "tol": 1e-8},
        # many dense symmetric eigenproblems of uneven size in one launch
        {"name": "batch_sym_512", "kind": "batch", "count": 512, "nmin": 64, "nmax": 1024, "nev": 8, "tol": 1e-7,
         "step": 6},
        # one Rayleigh-Ritz step on a 64-column block of a 3-D Laplacian, FP64 (the call's default arithmetic)
        {"name": "eig_rr_48c_b64_f64", "kind": "eig_rr", "nx": 48, "ny": 49, "nz": 50, "b": 64, "prec": "double"},
        # one Rayleigh-Ritz step of an SVD block, dense operator, FP64
        {"name": "svd_rr_4096x1024_b32_f64", "kind": "svd_rr", "m": 4096, "n": 1024, "b": 32, "prec": "double"},
        # the basis build of the 16-bit phase: 64 columns of 8192 rows, half storage, FP32 arithmetic
        {"name": "hess_half_8192x64", "kind": "basis", "orth": "hessenberg", "m": 8192, "n": 64, "pc": "single",
         "po": "half"},
        # the same basis in the reference's default precision
        {"name": "hess_double_8192x64", "kind": "basis", "orth": "hessenberg", "m": 8192, "n": 64, "pc": "double",
         "po": "double"},
        # the reference's default basis (modified Gram-Schmidt with re-orthogonalisation) of the same block
        {"name": "mgs_double_8192x64", "kind": "basis", "orth": "mgs", "m": 8192, "n": 64, "pc": "double",
         "po": "double"},
        # block operator product of the largest sparse operator, FP32: 2.1 million rows, 32 right-hand sides
        {"name": "csrmm_n_f32_128c_32", "kind": "csrmm", "nx": 128, "ny": 128, "nz": 128, "nrhs": 32, "trans": "N",
         "pc": "single", "pin": "single"},
        # transposed block operator product (the A'U of a sparse SVD), FP64
        {"name": "csrmm_t_f64_64c_16", "kind": "csrmm", "nx": 64, "ny": 64, "nz": 64, "nrhs": 16, "trans": "T",
         "pc": "double", "pin": "double"},
        # the dense 16-bit block product A V of a power step (K-contiguous operands, FP32 accumulation)
        {"name": "gemm_half_8192x64x2048", "kind": "gemm", "M": 8192, "N": 64, "K": 2048, "pin": "half",
         "po": "single"},
    ]


def _log_int(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    kind = rng.choice(["si_eig", "svd_mixed", "krylov", "batch", "eig_rr", "svd_rr", "hess", "gs", "lu", "csrmm", "csrmm",
                       "gemm"])
    if kind == "si_eig":
        k = rng.randint(4, 48)
        if rng.random() < 0.5:
            nx = _log_int(rng, 16, 300)
            dims = (nx, nx + 1, 1)
        else:
            nx = _log_int(rng, 8, 44)
            dims = (nx, nx + 1, nx + 2)
        return {"kind": kind, "nx": dims[0], "ny": dims[1], "nz": dims[2], "k": k, "maxiter": rng.randint(3, 8),
                "step": rng.randint(1, 4)}
    if kind == "svd_mixed":
        m = _log_int(rng, 512, 16384)
        n = rng.randint(m // 8, m // 4)
        nev = rng.randint(4, min(64, n // 4))
        return {"kind": kind, "m": m, "n": n, "block": max(nev + 16, int(1.5 * nev)), "nev": nev, "step": 6, "step64": 12,
                "tol": rng.choice([1e-6, 1e-8]), "factors": rng.choice(["dense", "reflectors"])}
    if kind == "krylov":
        return {"kind": kind, "n1": _log_int(rng, 16, 64), "nev": rng.randint(6, 20), "kdim": rng.choice([40, 48, 63, 64]),
                "mode": rng.choice(["mixed", "mixed", "fp64"]), "tol": 1e-8}
    if kind == "batch":
        return {"kind": kind, "count": _log_int(rng, 16, 512), "nmin": rng.choice([64, 64, 200]),
                "nmax": rng.choice([256, 511, 1024]), "nev": 8, "tol": 1e-7, "step": rng.choice([4, 6, 8])}
    if kind == "eig_rr":
        nx = _log_int(rng, 12, 60)
        return {"kind": kind, "nx": nx, "ny": nx + 1, "nz": nx + 2, "b": rng.randint(6, 110),
                "prec": rng.choice(["double", "single"])}
    if kind == "svd_rr":
        m = _log_int(rng, 600, 8192)
        n = rng.randint(m // 8, m // 4)
        return {"kind": kind, "m": m, "n": n, "b": rng.randint(4, 64), "prec": rng.choice(["double", "single"])}
    if kind in ("hess", "lu"):
        pc, po = rng.choice([("single", "half"), ("single", "single"), ("double", "double"), ("single", "bfloat16")])
        return {"kind": "basis", "orth": {"hess": "hessenberg", "lu": "lu"}[kind],
                "m": _log_int(rng, 300, 262144 if kind == "hess" else 30000),
                "n": rng.randint(5, 128 if kind == "hess" else 64), "pc": pc, "po": po}
    if kind == "gs":
        return {"kind": "basis", "orth": rng.choice(["mgs", "cgs"]), "m": _log_int(rng, 300, 100000),
                "n": rng.randint(5, 80), "pc": "double", "po": "double"}
    if kind == "csrmm":
        nx = _log_int(rng, 12, 128)
        pc, pin = rng.choice([("single", "single"), ("double", "double"), ("single", "half")])
        return {"kind": kind, "nx": nx, "ny": max(8, nx - rng.randint(0, 5)), "nz": rng.choice([1, nx, nx]),
                "nrhs": rng.choice([1, 3, 8, 16, 21, 32]), "trans": rng.choice(["N", "N", "T"]), "pc": pc, "pin": pin}
    pin = rng.choice(["half", "bfloat16"])
    return {"kind": "gemm", "M": _log_int(rng, 64, 16384), "N": rng.choice([16, 21, 32, 64, 65, 96, 128]),
            "K": _log_int(rng, 64, 8192), "pin": pin, "po": rng.choice(["single", pin])}


# ---- inputs ---------------------------------------------------------------------------------------------
def _gen(seed):
    api.context()  # the library's stream becomes torch's current one
    return torch.Generator(device="cuda").manual_seed(int(seed) % (1 << 62))


def _cm(x):
    """The same matrix stored column-major."""
    return x.t().contiguous().t()


def _stencil(case, g):
    """Centre, lower and upper coefficients per direction (x fastest): the Dirichlet Laplacian, or the
    convection-diffusion operator (Pe drawn from the seed) for the nonsymmetric kinds."""
    dims = (case["nx"], case["ny"], case["nz"]) if "nx" in case else (case["n1"],) * 3
    act = [d for d in dims if d > 1]
    if case["kind"] in ("si_eig", "eig_rr"):
        return dims, 2.0 * len(act), [(-1.0, -1.0)] * 3
    pe = 8.0 + 4.0 * float(torch.rand(1, generator=g, device="cuda", dtype=F64))
    co, c0 = [], 0.0
    for d, w in zip(dims, (1.0, 0.5, 0.25)):
        h = 1.0 / (d + 1)
        c = pe * w / (2 * h)
        co.append((-1.0 / h ** 2 - c, -1.0 / h ** 2 + c))
        c0 += 2.0 / h ** 2 if d > 1 else 0.0
    return dims, c0, co


def _csr(dims, c0, co, symmetric):
    nx, ny, nz = dims
    n = nx * ny * nz
    r = torch.arange(n, device="cuda")
    x, y, z = r % nx, (r // nx) % ny, r // (nx * ny)
    cols = [(r - nx * ny, z > 0, co[2][0]), (r - nx, y > 0, co[1][0]), (r - 1, x > 0, co[0][0]), (r, r >= 0, c0),
            (r + 1, x < nx - 1, co[0][1]), (r + nx, y < ny - 1, co[1][1]), (r + nx * ny, z < nz - 1, co[2][1])]
    mask = torch.stack([m for _, m, _ in cols], 1)
    idx = torch.stack([c for c, _, _ in cols], 1)[mask].to(torch.int32)
    val = torch.tensor([v for _, _, v in cols], device="cuda", dtype=F64).expand(n, 7)[mask].contiguous()
    ptr = torch.zeros(n + 1, dtype=torch.int32, device="cuda")
    ptr[1:] = torch.cumsum(mask.sum(1), 0).to(torch.int32)
    return api.CsrMatrix.from_device(ptr, idx, val, (n, n), symmetric=symmetric)


def _apply(dims, c0, co, X, trans=False):
    """The stencil times a block, in 64 bits."""
    nx, ny, nz = dims
    T = X.to(F64).t().reshape(-1, nz, ny, nx)
    Y = c0 * T
    for ax, (lo, up) in ((3, co[0]), (2, co[1]), (1, co[2])):
        L = T.shape[ax]
        if L < 2:
            continue
        if trans:
            lo, up = up, lo
        Y.narrow(ax, 1, L - 1).add_(T.narrow(ax, 0, L - 1), alpha=lo)
        Y.narrow(ax, 0, L - 1).add_(T.narrow(ax, 1, L - 1), alpha=up)
    return Y.reshape(X.shape[1], -1).t()


def _unit_max(X):
    """Columns scaled so that the largest entry is 1, as a power step leaves them."""
    k = X.abs().argmax(0)
    return X / X.gather(0, k[None, :])


def _reflect(X, W):
    """Products of Householder reflectors (rows of W) applied to the rows' space of X (in place)."""
    for w in W:
        X -= torch.outer(w, (2.0 / (w @ w)) * (w @ X))
    return X


def _mix(X, g):
    """A dense random orthogonal factor times X: random signs and Hartley transforms, three times."""
    N = X.shape[0]
    for _ in range(3):
        sign = torch.randint(0, 2, (N, 1), generator=g, device="cuda").to(F64) * 2 - 1
        f = torch.fft.fft(X * sign, dim=0)
        X = (f.real - f.imag) / math.sqrt(N)
    return X


def _spectrum_matrix(m, n, s, g, factors):
    """m x n with singular values s; the orthogonal factors dense ("dense") or products of three Householder
    reflectors ("reflectors", the serving stream's matrices)."""
    A = torch.zeros(m, n, dtype=F64, device="cuda")
    A[torch.arange(n), torch.arange(n)] = s
    if factors == "dense":
        return _mix(_mix(A, g).t(), g).t()
    A = _reflect(A, torch.randn(3, m, generator=g, device="cuda", dtype=F64))
    return _reflect(A.t().contiguous(), torch.randn(3, n, generator=g, device="cuda", dtype=F64)).t()


def _geometric(n):
    return 1e-6 ** (torch.arange(n, dtype=F64, device="cuda") / max(n - 1, 1))


def _batch_sizes(case, seed):
    """The matrices' sizes (the case's own) and spectra (the seed's)."""
    ns = np.random.default_rng(case["count"]).integers(case["nmin"], case["nmax"] + 1, case["count"]).astype(np.int64)
    rng = np.random.default_rng(int(seed))
    lams = [np.sort(np.exp(np.log(1e-4) * rng.random(int(n))))[::-1].copy() for n in ns]
    return ns, lams


def prepare(case, seed):
    kind = case["kind"]
    g = _gen(seed)
    randn = lambda *s: torch.randn(*s, generator=g, device="cuda", dtype=F64)  # noqa: E731
    st = {"case": case}
    if kind in ("si_eig", "krylov", "eig_rr", "csrmm"):
        dims, c0, co = _stencil(case, g)
        n = dims[0] * dims[1] * dims[2]
        st["A"] = _csr(dims, c0, co, kind in ("si_eig", "eig_rr"))
        if kind == "si_eig":
            st["V0"] = _cm(randn(n, case["k"]))
        elif kind == "krylov":
            st["v0"] = _cm(randn(n, 1))
        elif kind == "eig_rr":  # a random block after four power steps
            V = randn(n, case["b"])
            for _ in range(4):
                V = _unit_max(_apply(dims, c0, co, V))
            st["V"] = _cm(V.to(TORCH[case["prec"]]))
        else:
            st["X"] = _cm(randn(n, case["nrhs"]).to(TORCH[case["pin"]]))
    elif kind == "svd_mixed":
        s = _geometric(case["n"])
        st["A"], st["V0"] = _cm(_spectrum_matrix(case["m"], case["n"], s, g, case["factors"])), _cm(randn(case["n"], case["block"]))
    elif kind == "svd_rr":  # bases after two power steps
        A = _cm(_spectrum_matrix(case["m"], case["n"], _geometric(case["n"]), g, "dense"))
        V = _unit_max(A.t() @ (A @ randn(case["n"], case["b"])))
        dt = TORCH[case["prec"]]
        st["A"], st["U"], st["V"] = _cm(A.to(dt)), _cm(_unit_max(A @ V).to(dt)), _cm(V.to(dt))
    elif kind == "batch":
        ns, lams = _batch_sizes(case, seed)
        st["ns"], st["offs"] = ns, np.concatenate([[0], np.cumsum(ns * ns)[:-1]]).astype(np.int64)
        buf = torch.empty(int((ns * ns).sum()), dtype=F64, device="cuda")
        for n, off, lam in zip(ns, st["offs"], lams):
            n = int(n)
            Q = torch.diag(torch.from_numpy(lam).cuda())
            W = randn(3, n)
            Q = _reflect(_reflect(Q, W).t().contiguous(), W)
            buf[int(off):int(off) + n * n] = (0.5 * (Q + Q.t())).reshape(-1)
        st["A"] = buf
    elif kind == "basis":  # a block as power steps leave it: leading directions shared by all columns
        m, n = case["m"], case["n"]
        r = min(m, n + 16)
        decay = 10.0 ** (-3.0 * torch.arange(r, dtype=F64, device="cuda") / r)
        X = _unit_max((randn(m, r) * decay[None, :]) @ randn(r, n))
        st["X"] = _cm(X.to(TORCH[case["po"]]))
    elif kind == "gemm":
        dt = TORCH[case["pin"]]
        st["A"] = _cm(randn(case["K"], case["M"]).mul_(0.05).to(dt))
        st["B"] = _cm(_unit_max(randn(case["K"], case["N"])).to(dt))
    else:
        raise ValueError(kind)
    return st


# ---- one pass -------------------------------------------------------------------------------------------
def run(st):
    c = st["case"]
    kind = c["kind"]
    if kind == "si_eig":
        A = st["A"]
        V, d, _ = api.subspace_iter_eig(A, A.shape[0], c["k"], "double", maxiter=c["maxiter"], step_size=c["step"],
                                        V0=st["V0"])
        return {"V": V, "d": d}
    if kind == "svd_mixed":
        U, s, V, _ = api.subspace_iter_svd(st["A"], c["m"], c["n"], c["block"], "single", "half", maxiter=80,
                                           step_size=c["step"], step_size_f64=c["step64"], V0=st["V0"], mode="mixed",
                                           tol=c["tol"], nev=c["nev"])
        return {"U": U, "s": s, "V": V}
    if kind == "krylov":
        A = st["A"]
        X, d, _ = api.arnoldi_hess_eig(A, A.shape[0], c["nev"], "single", "half" if c["mode"] == "mixed" else None,
                                       maxiter=40000, kdim=c["kdim"], v0=st["v0"], mode=c["mode"], tol=c["tol"])
        return {"X": X, "d": d}
    if kind == "batch":
        Xs, ev, _, _, sts = api.batch_sym_eig(st["A"], st["ns"], st["offs"], nev=c["nev"], tol=c["tol"],
                                              step_size=c["step"])
        return {"X": Xs[0]._base, "ev": ev, "status": sts}  # every vector: the matrices' X are views of one tensor
    if kind == "eig_rr":
        V, d = api.eig_rr(st["A"], st["V"], c["prec"], use_generalized=True)
        return {"V": V, "d": d}
    if kind == "svd_rr":
        U, s, V = api.svd_rr(st["A"], st["U"], st["V"], c["prec"])
        return {"U": U, "s": s, "V": V}
    if kind == "basis":
        if c["orth"] == "hessenberg":
            Q, R, sel, perm = api.hessenberg(st["X"], c["pc"], c["po"])
            return {"Q": Q, "R": R, "select": sel.astype(np.int64), "perm": perm}
        if c["orth"] == "lu":
            Q, R, skip = api.lu_basis(st["X"], c["pc"], c["po"])
        else:
            Q, R, skip = api.gs_basis(st["X"], c["orth"] == "cgs", c["pc"], c["po"])
        return {"Q": Q, "R": R, "skip": skip}
    if kind == "csrmm":
        return {"Y": api.csrmv(st["A"], c["trans"], st["X"], c["pc"])}
    return {"C": api.gemm(st["A"], "T", st["B"], "single", c["po"])}


# ---- what a pass cannot do without ------------------------------------------------------------------------
def work(case):
    c = case
    kind = c["kind"]
    if kind in ("si_eig", "krylov", "eig_rr", "csrmm"):
        nx, ny, nz = (c["nx"], c["ny"], c["nz"]) if "nx" in c else (c["n1"],) * 3
        n = nx * ny * nz
        nnz = n + 2 * (n // nx * (nx - 1) + n // ny * (ny - 1) + n // nz * (nz - 1))
        mat = 4.0 * (nnz + n)
    if kind == "si_eig":
        b = c["k"]
        per = 2.0 * nnz * b * (c["step"] + 1) + n * b * b * (1 + 3 * 2)
        return {"bytes": mat + 8.0 * nnz + 16.0 * n * b, "flops": c["maxiter"] * per}
    if kind == "svd_mixed":
        m, n, b = c["m"], c["n"], c["block"]
        # power steps that the spectrum asks for: (s_{b+1} / s_nev)^(2 steps) below the tolerance
        gap = math.log(1e6) * (b + 1 - c["nev"]) / max(n - 1, 1)
        steps = math.ceil(-math.log(c["tol"]) / (2 * gap))
        return {"bytes": 8.0 * m * n + 8.0 * b * (m + 2 * n), "flops": 4.0 * m * n * b * steps}
    if kind == "krylov":
        nb, keep = c["kdim"] + 1, c["nev"]
        # one cycle at least: the steps with their eliminations, the block product, two Gram matrices
        return {"bytes": mat + 8.0 * nnz + 8.0 * n * (1 + keep),
                "flops": 2.0 * nnz * nb * 2 + n * nb * nb * (1 + 2 + 2) + 2.0 * n * nb * keep}
    if kind == "batch":
        mean_sq = (c["nmin"] ** 2 + c["nmin"] * c["nmax"] + c["nmax"] ** 2) / 3.0
        mean = 0.5 * (c["nmin"] + c["nmax"])
        return {"bytes": c["count"] * 8.0 * (mean_sq + c["nev"] * mean),
                "flops": c["count"] * 2.0 * mean_sq * 16 * 4 * c["step"]}
    if kind == "eig_rr":
        b, e = c["b"], BYTES[c["prec"]]
        return {"bytes": mat + e * (nnz + 2.0 * n * b), "flops": 2.0 * nnz * b + 6.0 * n * b * b}
    if kind == "svd_rr":
        m, n, b, e = c["m"], c["n"], c["b"], BYTES[c["prec"]]
        return {"bytes": e * (m * n + 2.0 * (m + n) * b), "flops": 2.0 * m * n * b + 2.0 * b * b * (3 * m + 2 * n)}
    if kind == "basis":
        m, n, e = c["m"], c["n"], BYTES[c["po"]]
        f = {"hessenberg": 1.0, "lu": 1.0, "mgs": 2.0, "cgs": 2.0}[c["orth"]]
        return {"bytes": 2.0 * m * n * e + 8.0 * n * n, "flops": f * m * n * n}
    if kind == "csrmm":
        e, v = BYTES[c["pin"]], BYTES[c["pc"]]
        return {"bytes": mat + v * nnz + (e + v) * float(n) * c["nrhs"], "flops": 2.0 * nnz * c["nrhs"]}
    M, N, K = c["M"], c["N"], c["K"]
    return {"bytes": 2.0 * K * (M + N) + BYTES[c["po"]] * float(M) * N, "flops": 2.0 * M * N * K}


# ---- the same results in 64 bits ---------------------------------------------------------------------------
def _gs_exact(X):
    """Modified Gram-Schmidt with the adaptive re-orthogonalisation, column by column."""
    m, n = X.shape
    Q, R = torch.zeros_like(X), torch.zeros(n, n, dtype=F64)
    for i in range(n):
        v = X[:, i].clone()
        norm = float(v.norm())
        t = None
        while t is None or (t >= 2.0 ** -52 and t < norm / math.sqrt(2.0)):
            norm = norm if t is None else t
            r = Q[:, :i].t() @ v
            v = v - Q[:, :i] @ r
            R[:i, i] += r.cpu()
            t = float(v.norm())
        Q[:, i] = v / t
        R[i, i] = t
    return Q, R


def _hess_exact(X):
    """Pivoted elimination: every column against the earlier ones, then divided by its largest entry."""
    W = X.clone()
    m, n = W.shape
    R, perm = torch.zeros(n, n, dtype=F64), torch.zeros(n, dtype=torch.int64)
    for j in range(n):
        k = int(W[:, j].abs().argmax())
        perm[j] = k
        R[j, j:] = W[k, j:].cpu()
        W[:, j] = W[:, j] / W[k, j].clone()
        W[:, j + 1:] -= torch.outer(W[:, j], W[k, j + 1:].clone())
    return W, R, perm


def exact(case, seed):
    c = case
    kind = c["kind"]
    if kind == "batch":
        _, lams = _batch_sizes(c, seed)
        return {"X": None, "ev": np.array([l[: c["nev"]] for l in lams]), "status": None}
    if kind == "svd_mixed":
        return {"U": None, "s": _geometric(c["n"])[: c["block"]], "V": None}
    if kind == "krylov":
        dims, _, co = _stencil(c, _gen(seed))
        parts = []
        for d, (lo, up) in zip(dims, co):
            k = torch.arange(1, d + 1, dtype=F64, device="cuda")
            parts.append(2.0 * (d + 1) ** 2 - 2.0 * math.sqrt(lo * up) * torch.cos(k * math.pi / (d + 1)))
        lam = (parts[0][:, None, None] + parts[1][None, :, None] + parts[2][None, None, :]).reshape(-1)
        return {"X": None, "d": torch.topk(lam, c["nev"]).values}
    st = prepare(c, seed)
    if kind == "si_eig":
        dims, c0, co = _stencil(c, _gen(seed))
        V = st["V0"]
        for _ in range(c["maxiter"]):
            for _ in range(c["step"]):
                V = _apply(dims, c0, co, V)
            V = torch.linalg.qr(V).Q
        d = torch.linalg.eigvalsh(V.t() @ _apply(dims, c0, co, V))
        return {"V": None, "d": d.flip(0)}
    if kind == "eig_rr":
        dims, c0, co = _stencil(c, _gen(seed))
        V = st["V"].to(F64)
        L = torch.linalg.cholesky(V.t() @ V + 1e-10 * torch.eye(c["b"], dtype=F64, device="cuda"))
        H = torch.linalg.solve_triangular(L, V.t() @ _apply(dims, c0, co, V), upper=False)
        H = torch.linalg.solve_triangular(L, H.t(), upper=False)
        return {"V": None, "d": torch.linalg.eigvalsh(0.5 * (H + H.t())).flip(0)}
    if kind == "svd_rr":
        A, U, V = st["A"].to(F64), st["U"].to(F64), st["V"].to(F64)
        I = 1e-10 * torch.eye(c["b"], dtype=F64, device="cuda")
        Lu, Lv = torch.linalg.cholesky(U.t() @ U + I), torch.linalg.cholesky(V.t() @ V + I)
        C = torch.linalg.solve_triangular(Lu, U.t() @ (A @ V), upper=False)
        C = torch.linalg.solve_triangular(Lv, C.t(), upper=False)
        return {"U": None, "s": torch.linalg.svdvals(C), "V": None}
    if kind == "basis":
        if c["po"] != "double":
            return None  # every entry is rounded to the storage type as the elimination goes on
        if c["orth"] == "hessenberg":
            Q, R, perm = _hess_exact(st["X"])
            return {"Q": Q, "R": R, "select": None, "perm": None}
        if c["orth"] == "lu":
            Q, R, perm = _hess_exact(st["X"])  # with every column kept, lu.m's two-output L and U are these
            return {"Q": Q, "R": R, "skip": None}
        Q, R = _gs_exact(st["X"])
        return {"Q": Q, "R": R, "skip": None}
    if kind == "csrmm":
        dims, c0, co = _stencil(c, _gen(seed))
        return {"Y": _apply(dims, c0, co, st["X"], c["trans"] == "T")}
    return {"C": st["A"].to(F64).t() @ st["B"].to(F64)}
