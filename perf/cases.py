"""Performance cases of the library: the calls its users make, with their sizes.

A case names an operation (`op`) and its sizes:

  chol       FLA_Chol of one SPD matrix (a copy of the pristine matrix, as a
             caller that keeps A makes it, then the factorization in place)
  lu         FLA_LU_piv of one general matrix, square or rectangular
  qr         FLA_QR_UT of one m x n matrix, m > n, T blocks of 32 columns
  apply_q    FLA_Apply_Q_UT of a kept QR factorization to a block of columns
  solve      FLA_LU_piv_solve / FLA_Chol_solve with a kept factorization
  mixed      FLA_B200_Chol_solve_mixed / FLA_B200_LU_piv_solve_mixed:
             low-precision factors with FP64 refinement, right-hand sides at once
  adjoint    FLA_Chol_adjoint of one factor (reverse mode)
  batched    FLA_Chol_batched / FLA_B200_Chol_batched_logdet /
             FLA_LU_piv_batched (+ the FP32 forms) of many small systems of
             different orders with their right-hand sides

Matrices are column-major; an odd leading dimension, which the device copies
behind the calls have to realign, occurs like any other.
"""
import ctypes as C
import math
import random

import numpy as np
import torch

import libflame_b200 as F

T_BLOCK = 32  # the interface's T block for QR_UT


def listed():
    return [
        # the headline factorizations: one dense system that fills a few GiB
        {"name": "lu_16384", "op": "lu", "m": 16384, "n": 16384},
        {"name": "chol_16384", "op": "chol", "n": 16384, "upper": False},
        # least squares at size: a tall matrix's orthogonal factorization
        {"name": "qr_12288x6144", "op": "qr", "m": 12288, "n": 6144},
        # everyday sizes: the reference's own CPU configuration, and an odd
        # order whose columns are not 16-byte aligned
        {"name": "chol_1024", "op": "chol", "n": 1024, "upper": False},
        {"name": "lu_3001", "op": "lu", "m": 3001, "n": 3001},
        # one small system: launches and waits are all there is
        {"name": "chol_100", "op": "chol", "n": 100, "upper": False},
        # a kept factorization used for new right-hand sides
        {"name": "lu_solve_8192x32", "op": "solve", "kind": "lu", "n": 8192, "nrhs": 32},
        {"name": "apply_q_8192x4096x64", "op": "apply_q", "m": 8192, "n": 4096, "nrhs": 64, "trans": True},
        # time to solution with low-precision factors
        {"name": "mixed_spd_8192x32", "op": "mixed", "kind": "spd", "n": 8192, "nrhs": 32, "kappa": 1e2},
        # reverse mode through a Cholesky (Gaussian-process training)
        {"name": "adjoint_4096", "op": "adjoint", "n": 4096},
        # many small systems of different orders, with four right-hand sides
        {"name": "batched_chol_2500", "op": "batched", "kind": "chol", "f32": False, "logdet": False, "count": 2500,
         "lo": 8, "hi": 512, "nrhs": 4},
        {"name": "batched_lu_2500", "op": "batched", "kind": "lu", "f32": False, "logdet": False, "count": 2500,
         "lo": 8, "hi": 512, "nrhs": 4},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    op = rng.choice(["chol", "chol", "lu", "lu", "qr", "apply_q", "solve", "mixed", "adjoint", "batched", "batched"])
    if op == "chol":
        return {"op": op, "n": _log_int(rng, 64, 16384), "upper": rng.random() < 0.25}
    if op == "lu":
        m = _log_int(rng, 64, 16384)
        n = m if rng.random() < 0.6 else _log_int(rng, 64, 16384)
        return {"op": op, "m": m, "n": n}
    if op == "qr":
        n = _log_int(rng, 32, 6144)
        return {"op": op, "m": n + _log_int(rng, 1, 6144), "n": n}
    if op == "apply_q":
        n = _log_int(rng, 64, 4096)
        return {"op": op, "m": n + _log_int(rng, 1, 4096), "n": n, "nrhs": _log_int(rng, 1, 512),
                "trans": rng.random() < 0.7}
    if op == "solve":
        return {"op": op, "kind": rng.choice(["lu", "chol"]), "n": _log_int(rng, 64, 8192), "nrhs": _log_int(rng, 1, 256)}
    if op == "mixed":
        return {"op": op, "kind": rng.choice(["spd", "general"]), "n": _log_int(rng, 256, 8192),
                "nrhs": _log_int(rng, 1, 64), "kappa": 10.0 ** rng.uniform(1.0, 4.0)}
    if op == "adjoint":
        return {"op": op, "n": _log_int(rng, 64, 4096)}
    kind = rng.choice(["chol", "chol", "lu"])
    logdet = kind == "chol" and rng.random() < 0.4
    lo = _log_int(rng, 8, 64)
    return {"op": op, "kind": kind, "f32": not logdet and rng.random() < 0.25, "logdet": logdet,
            "count": _log_int(rng, 32, 2500), "lo": lo, "hi": _log_int(rng, 64, 512) if not logdet else
            _log_int(rng, 64, 768), "nrhs": 1 if logdet else rng.choice([0, 1, 4, 7])}


# ---------------------------------------------------------------------------
# Inputs.
# ---------------------------------------------------------------------------
def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed))


def _empty(m, n, dtype=torch.float64):
    return torch.empty_strided((m, n), (1, max(m, 1)), dtype=dtype, device="cuda")


def _colmajor(t):
    out = _empty(t.shape[0], t.shape[1], t.dtype)
    out.copy_(t)
    return out


def _randn(m, n, g):
    return torch.randn((n, m), dtype=torch.float64, device="cuda", generator=g).t()


def _uniform(m, n, g):
    return torch.rand((n, m), dtype=torch.float64, device="cuda", generator=g).mul_(2).sub_(1).t()


def _spd(n, g):
    """G G^T / n + I, G of N(0,1) entries."""
    G = torch.randn((n, n), dtype=torch.float64, device="cuda", generator=g)
    A = G @ G.t()
    A.div_(n).diagonal().add_(1.0)
    return A.t()


def _with_kappa(kind, n, kappa, g):
    """Q diag(s) Q^T (spd) or Q diag(s) V^T, s log-spaced from 1 to 1 / kappa."""
    Q = torch.linalg.qr(torch.randn((n, n), dtype=torch.float64, device="cuda", generator=g))[0]
    V = Q if kind == "spd" else torch.linalg.qr(torch.randn((n, n), dtype=torch.float64, device="cuda", generator=g))[0]
    s = torch.logspace(0, -math.log10(kappa), n, dtype=torch.float64, device="cuda")
    A = (Q * s) @ V.t()
    if kind == "spd":
        A = (A + A.t()) / 2
    return _colmajor(A)


def _batch_sizes(case):
    """The batch's orders: the case's own, whatever the entries' seed."""
    r = random.Random(case["count"])
    lo, hi = min(case["lo"], case["hi"]), max(case["lo"], case["hi"])
    return np.array([r.randint(lo, hi) for _ in range(case["count"])], dtype=np.int64)


def _batch_inputs(case, seed):
    """Orders, offsets and the two flat buffers (column-major matrices and
    right-hand sides one after another)."""
    sizes = _batch_sizes(case)
    g = _gen(seed)
    dt = torch.float32 if case["f32"] else torch.float64
    offs = np.concatenate([[0], np.cumsum(sizes ** 2)])
    boffs = np.concatenate([[0], np.cumsum(sizes * case["nrhs"])])
    src = torch.empty(int(offs[-1]), dtype=dt, device="cuda")
    for nv in np.unique(sizes):
        idx = np.nonzero(sizes == nv)[0]
        nv = int(nv)
        if case["kind"] == "chol":
            G = torch.randn((len(idx), nv, nv), dtype=torch.float64, device="cuda", generator=g)
            M = G @ G.transpose(1, 2) / nv + torch.eye(nv, dtype=torch.float64, device="cuda")
        else:
            M = torch.rand((len(idx), nv, nv), dtype=torch.float64, device="cuda", generator=g) * 2 - 1
        for q, i in enumerate(idx):
            src[int(offs[i]):int(offs[i + 1])] = M[q].reshape(-1).to(dt)  # column-major: the transpose's rows
    rhs = torch.randn(max(1, int(boffs[-1])), dtype=torch.float64, device="cuda", generator=g).to(dt)
    return sizes, offs, boffs, src, rhs


def prepare(case, seed):
    F.init()
    op, g = case["op"], _gen(seed)
    if op == "chol":
        A0 = _spd(case["n"], g)
        return {"case": case, "A0": A0, "A": torch.empty_like(A0)}
    if op == "lu":
        A0 = _uniform(case["m"], case["n"], g)
        p = torch.zeros(min(case["m"], case["n"]), dtype=torch.int32, device="cuda")
        return {"case": case, "A0": A0, "A": torch.empty_like(A0), "p": p}
    if op == "qr":
        A0 = _randn(case["m"], case["n"], g)
        T = _colmajor(torch.zeros((min(T_BLOCK, case["n"]), case["n"]), dtype=torch.float64, device="cuda"))
        return {"case": case, "A0": A0, "A": torch.empty_like(A0), "T": T}
    if op == "apply_q":
        A = _randn(case["m"], case["n"], g)
        T = _colmajor(torch.zeros((min(T_BLOCK, case["n"]), case["n"]), dtype=torch.float64, device="cuda"))
        B0 = _randn(case["m"], case["nrhs"], g)
        _done(F.qr_ut(A, T))
        return {"case": case, "A": A, "T": T, "B0": B0, "B": torch.empty_like(B0)}
    if op == "solve":
        n = case["n"]
        A = _uniform(n, n, g) if case["kind"] == "lu" else _spd(n, g)
        B = _randn(n, case["nrhs"], g)
        p = torch.zeros(n, dtype=torch.int32, device="cuda")
        _done(F.lu_piv(A, p) if case["kind"] == "lu" else F.chol(A))
        return {"case": case, "A": A, "p": p, "B": B, "X": torch.empty_like(B)}
    if op == "mixed":
        A = _with_kappa(case["kind"], case["n"], case["kappa"], g)
        B = _randn(case["n"], case["nrhs"], g)
        return {"case": case, "A": A, "B": B, "X": torch.empty_like(B)}
    if op == "adjoint":
        n = case["n"]
        L = _colmajor(torch.linalg.cholesky(_spd(n, g)))
        Lbar0 = _colmajor(torch.tril(_randn(n, n, g)))
        return {"case": case, "L": L, "Lbar0": Lbar0, "Lbar": torch.empty_like(Lbar0)}
    sizes, offs, boffs, src, rhs = _batch_inputs(case, seed)
    work, bwork = src.clone(), rhs.clone()
    count, es = case["count"], src.element_size()
    poffs = np.concatenate([[0], np.cumsum(sizes)])
    piv = torch.zeros(int(sizes.sum()), dtype=torch.int32, device="cuda")
    ptrs = lambda base, o, w: (C.c_void_p * count)(*[base + int(o[i]) * w for i in range(count)])  # noqa: E731
    return {"case": case, "src": src, "rhs": rhs, "work": work, "bwork": bwork, "piv": piv,
            "n": sizes.astype(np.int32), "A": ptrs(work.data_ptr(), offs, es), "B": ptrs(bwork.data_ptr(), boffs, es),
            "P": ptrs(piv.data_ptr(), poffs, 4), "info": np.zeros(count, dtype=np.int32),
            "logdet": np.zeros(count, dtype=np.float64)}


def _done(r):
    if r != F.FLA_SUCCESS:
        raise RuntimeError("call returned %d: %s" % (r, F.last_error()))


# ---------------------------------------------------------------------------
# One pass.
# ---------------------------------------------------------------------------
def run(state):
    case = state["case"]
    op = case["op"]
    if op == "chol":
        state["A"].copy_(state["A0"])
        _done(F.chol(state["A"], F.FLA_UPPER_TRIANGULAR if case["upper"] else F.FLA_LOWER_TRIANGULAR))
        return state["A"]
    if op == "lu":
        state["A"].copy_(state["A0"])
        _done(F.lu_piv(state["A"], state["p"]))
        return state["A"], state["p"]
    if op == "qr":
        state["A"].copy_(state["A0"])
        _done(F.qr_ut(state["A"], state["T"]))
        return state["A"], state["T"]
    if op == "apply_q":
        state["B"].copy_(state["B0"])
        _done(F.apply_q_ut(state["A"], state["T"], state["B"],
                           F.FLA_CONJ_TRANSPOSE if case["trans"] else F.FLA_NO_TRANSPOSE))
        return state["B"]
    if op == "solve":
        if case["kind"] == "lu":
            _done(F.lu_piv_solve(state["A"], state["p"], state["B"], state["X"]))
        else:
            _done(F.chol_solve(state["A"], state["B"], state["X"]))
        return state["X"]
    if op == "mixed":
        f = F.chol_solve_mixed if case["kind"] == "spd" else F.lu_piv_solve_mixed
        _done(f(state["A"], state["B"], state["X"])[0])
        return state["X"]
    if op == "adjoint":
        state["Lbar"].copy_(state["Lbar0"])
        _done(F.chol_adjoint(state["L"], state["Lbar"]))
        return state["Lbar"]
    return _run_batched(state, case)


def _run_batched(s, case):
    lib, count, nrhs = F.lib(), case["count"], case["nrhs"]
    P = lambda a: a.ctypes.data_as(C.c_void_p)  # noqa: E731
    s["work"].copy_(s["src"])
    s["bwork"].copy_(s["rhs"])
    n, info = P(s["n"]), P(s["info"])
    B, ldb = (s["B"], n) if nrhs else (None, None)
    if case["logdet"]:
        _done(lib.FLA_B200_Chol_batched_logdet(count, n, s["A"], n, nrhs, B, ldb, P(s["logdet"]), info))
        return s["work"], s["bwork"], s["logdet"], s["info"]
    if case["kind"] == "chol":
        if case["f32"]:
            _done(lib.FLA_B200_Chol_batched_f32(count, n, s["A"], n, nrhs, B, ldb, info))
        else:
            _done(lib.FLA_Chol_batched(F.FLA_LOWER_TRIANGULAR, count, n, s["A"], n, nrhs, B, ldb, info))
        return s["work"], s["bwork"], s["info"]
    f = lib.FLA_B200_LU_piv_batched_f32 if case["f32"] else lib.FLA_LU_piv_batched
    _done(f(count, n, s["A"], n, s["P"], nrhs, B, ldb, info))
    return s["work"], s["bwork"], s["piv"], s["info"]


# ---------------------------------------------------------------------------
# The work of one pass: inputs read once, outputs written once.
# ---------------------------------------------------------------------------
def work(case):
    op = case["op"]
    if op == "chol":
        n = case["n"]  # one triangle read, one written
        return {"bytes": 8.0 * n * (n + 1), "flops": n ** 3 / 3.0}
    if op == "lu":
        m, n = case["m"], case["n"]
        k = min(m, n)
        return {"bytes": 16.0 * m * n + 4.0 * k, "flops": 2.0 * m * n * k - (m + n) * float(k) * k + 2.0 * k ** 3 / 3}
    if op == "qr":
        m, n = case["m"], case["n"]
        return {"bytes": 16.0 * m * n + 8.0 * T_BLOCK * n, "flops": 2.0 * m * n * n - 2.0 * n ** 3 / 3}
    if op == "apply_q":
        m, n, r = case["m"], case["n"], case["nrhs"]
        return {"bytes": 8.0 * (m * n - n * n / 2.0) + 16.0 * m * r, "flops": 4.0 * m * n * r - 2.0 * n * n * r}
    if op == "solve":
        n, r = case["n"], case["nrhs"]
        return {"bytes": 8.0 * n * n * (1.0 if case["kind"] == "lu" else 0.5) + 16.0 * n * r, "flops": 2.0 * n * n * r}
    if op == "mixed":
        n, r = case["n"], case["nrhs"]
        spd = case["kind"] == "spd"
        return {"bytes": 8.0 * n * n * (0.5 if spd else 1.0) + 16.0 * n * r,
                "flops": n ** 3 * (1.0 if spd else 2.0) / 3 + 2.0 * n * n * r}
    if op == "adjoint":
        n = case["n"]  # L and Lbar read, Abar written: one triangle each
        return {"bytes": 12.0 * n * (n + 1), "flops": 2.0 * n ** 3 / 3}
    # orders uniform between the two bounds: means of n^2 and n^3
    lo, hi = min(case["lo"], case["hi"]), max(case["lo"], case["hi"])
    v = np.arange(lo, hi + 1, dtype=np.float64)
    es = 4.0 if case["f32"] else 8.0
    tri = case["kind"] == "chol"
    byt = case["count"] * es * (np.mean(v ** 2) * (1.0 if tri else 2.0) + 2.0 * case["nrhs"] * np.mean(v))
    flo = case["count"] * (np.mean(v ** 3) * (1.0 if tri else 2.0) / 3 + 2.0 * case["nrhs"] * np.mean(v ** 2))
    return {"bytes": float(byt), "flops": float(flo)}


# ---------------------------------------------------------------------------
# The same results from torch in 64 bits.
# ---------------------------------------------------------------------------
def _relative(piv):
    """LAPACK's 1-based pivot rows as the interface's offsets from the column."""
    return (piv - 1 - torch.arange(piv.shape[-1], device=piv.device, dtype=piv.dtype)).to(torch.int32)


def _chol_in_place(A, upper):
    """The factor in its triangle, the other triangle as it was."""
    L = torch.linalg.cholesky(A)
    return torch.triu(L.t()) + torch.tril(A, -1) if upper else torch.tril(L) + torch.triu(A, 1)


def _qr_t(QR, n):
    """T: striu(V^T V) + diag(V^T V) / 2 for each block of T_BLOCK columns."""
    b = min(T_BLOCK, n)
    T = torch.zeros((b, n), dtype=torch.float64, device=QR.device)
    for j in range(0, n, b):
        w = min(b, n - j)
        V = torch.tril(QR[j:, j:j + w], -1)
        V[:w].diagonal().fill_(1.0)
        G = V.t() @ V
        T[:w, j:j + w] = torch.triu(G, 1) + torch.diag(G.diagonal() / 2)
    return T


def exact(case, seed):
    op, g = case["op"], _gen(seed)
    if op == "chol":
        return _chol_in_place(_spd(case["n"], g), case["upper"])
    if op == "lu":
        return torch.linalg.lu_factor(_uniform(case["m"], case["n"], g))[0], None
    if op == "qr":
        QR = torch.geqrf(_randn(case["m"], case["n"], g))[0]
        return QR, _qr_t(QR, case["n"])
    if op == "apply_q":
        QR, tau = torch.geqrf(_randn(case["m"], case["n"], g))
        B = _randn(case["m"], case["nrhs"], g)
        return torch.ormqr(QR, tau, B, left=True, transpose=case["trans"])
    if op in ("solve", "mixed"):
        n = case["n"]
        if op == "mixed":
            A = _with_kappa(case["kind"], n, case["kappa"], g)
        else:
            A = _uniform(n, n, g) if case["kind"] == "lu" else _spd(n, g)
        return torch.linalg.solve(A, _randn(n, case["nrhs"], g))
    if op == "adjoint":
        n = case["n"]
        L = torch.linalg.cholesky(_spd(n, g))
        P = torch.tril(L.t() @ torch.tril(_randn(n, n, g)))
        P.diagonal().mul_(0.5)
        Li = torch.linalg.solve_triangular(L, torch.eye(n, dtype=torch.float64, device="cuda"), upper=False)
        S = Li.t() @ (P + P.t()) @ Li  # the gradient by the lower entries alone
        S.diagonal().mul_(0.5)
        return torch.tril(S)
    return _exact_batched(case, seed)


def _exact_batched(case, seed):
    sizes, offs, boffs, src, rhs = _batch_inputs(case, seed)
    src, rhs, r = src.double(), rhs.double(), case["nrhs"]
    out, sol = src.clone(), rhs.clone()
    logdet = np.zeros(case["count"], dtype=np.float64)
    for nv in np.unique(sizes):
        idx = np.nonzero(sizes == nv)[0]
        nv = int(nv)
        M = torch.stack([src[int(offs[i]):int(offs[i + 1])].view(nv, nv).t() for i in idx])
        if case["kind"] == "chol":
            L = torch.linalg.cholesky(M)
            R = torch.tril(L) + torch.triu(M, 1)
            logdet[idx] = torch.log(L.diagonal(dim1=1, dim2=2)).sum(1).cpu().numpy()
        else:
            R = torch.linalg.lu_factor(M)[0]
        if r:
            B = torch.stack([rhs[int(boffs[i]):int(boffs[i + 1])].view(r, nv).t() for i in idx])
            X = torch.linalg.solve(M, B)
        for q, i in enumerate(idx):
            out[int(offs[i]):int(offs[i + 1])] = R[q].t().reshape(-1)
            if r:
                sol[int(boffs[i]):int(boffs[i + 1])] = X[q].t().reshape(-1)
    if case["logdet"]:
        return out, sol, logdet, None
    return (out, sol, None) if case["kind"] == "chol" else (out, sol, None, None)
