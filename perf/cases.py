"""The work that a program has this library do, as cases that can be timed and compared.

Every case is one pass through the public entry points on device data that is laid out once:

* gemm: the matched-order product `gemm_`, plain (C = A B) or as an update (C = C0 - A B, the
  form a blocked algorithm or a residual uses), from a few dozen rows to above a thousand;
* gemv: the matched-order matrix-vector product, both orientations;
* int8: the INT8 tensor-core product of operands with a wide exponent spread;
* chol, lu, ldlt: factor a copy of the matrix and solve for the right-hand sides;
* rrqr: rank-revealing QR and the least-squares solution;
* mixed_lu: the binary64 factor with refinement to full Float64xN accuracy;
* spd_batch: many uneven SPD blocks, factored, solved and differentiated.

Inputs and the exact values are made with plain torch: a multi-limb value is a list of float64
tensors, and products are sums of exact float64 matrix products of short slices.
"""
from __future__ import annotations

import importlib.util
import math
import os
import sys

import numpy as np
import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
PACKAGE = "mflab200"


def _package():
    """The package (its folder's name is not a Python identifier)."""
    if PACKAGE not in sys.modules:
        folder = os.path.join(ROOT, "multifloatlinearalgebra.jl_b200")
        spec = importlib.util.spec_from_file_location(
            PACKAGE, os.path.join(folder, "__init__.py"), submodule_search_locations=[folder])
        sys.modules[PACKAGE] = module = importlib.util.module_from_spec(spec)
        spec.loader.exec_module(module)
    return sys.modules[PACKAGE]


# ------------------------------------------------------------------ cases ----
def listed():
    return [
        # a small dense product inside a host loop (a panel, a small constraint block): the
        # time of one launch
        {"name": "gemm_x2_small", "kind": "gemm", "limbs": 2, "m": 48, "k": 40, "n": 56,
         "update": False},
        # the ordinary Float64x2 product at n = 256
        {"name": "gemm_x2_256", "kind": "gemm", "limbs": 2, "m": 256, "k": 256, "n": 256,
         "update": False},
        # a ragged Float64x4 update, as a blocked algorithm over uneven blocks issues it
        {"name": "gemm_x4_ragged", "kind": "gemm", "limbs": 4, "m": 515, "k": 389, "n": 777,
         "update": True},
        # a matrix-vector product of an iterative method or of a refinement step
        {"name": "gemv_x2", "kind": "gemv", "limbs": 2, "m": 2500, "n": 3100, "trans": "N"},
        # a ragged Float64x4 product on the tensor-core route
        {"name": "int8_x4_ragged", "kind": "int8", "limbs": 4, "m": 1531, "k": 2049, "n": 1203},
        # the large Float64x2 product on the tensor-core route
        {"name": "int8_x2_8192", "kind": "int8", "limbs": 2, "m": 8192, "k": 8192, "n": 8192},
        # Cholesky at n = 2048 with 64 right-hand sides
        {"name": "chol_x2_2048", "kind": "chol", "limbs": 2, "n": 2048, "rhs": 64},
        # a general Float64x4 system of ordinary, odd size
        {"name": "lu_x4_701", "kind": "lu", "limbs": 4, "n": 701, "rhs": 16},
        # a symmetric indefinite (saddle point) Float64x3 system
        {"name": "ldlt_x3_600", "kind": "ldlt", "limbs": 3, "n": 600, "rhs": 5},
        # least squares on a tall panel with the numerical rank
        {"name": "rrqr_x2_500x40", "kind": "rrqr", "limbs": 2, "m": 500, "n": 40, "rhs": 3},
        # the ill-conditioned Float64x4 system at n = 4096, solved by refinement
        {"name": "mixed_lu_x4_4096", "kind": "mixed_lu", "limbs": 4, "n": 4096, "rhs": 16,
         "decades": 12},
        # ten thousand SPD blocks of 8 to 256 rows with the gradients of the solution
        {"name": "spd_batch_10000", "kind": "spd_batch", "limbs": 2, "blocks": 10000, "least": 8,
         "most": 256},
    ]


def draw(rng):
    def size(low, high):
        return int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))

    kind = rng.choice(["gemm", "gemm", "gemv", "int8", "chol", "lu", "ldlt", "rrqr", "mixed_lu",
                       "spd_batch"])
    N = rng.choice([2, 3, 4])
    if kind == "gemm":
        return {"kind": kind, "limbs": N, "m": size(16, 1500), "k": size(16, 1500),
                "n": size(16, 1500), "update": rng.random() < 0.5}
    if kind == "gemv":
        return {"kind": kind, "limbs": N, "m": size(64, 4096), "n": size(64, 4096),
                "trans": rng.choice(["N", "T"])}
    if kind == "int8":
        return {"kind": kind, "limbs": N, "m": size(256, 5000), "k": size(256, 5000),
                "n": size(256, 5000)}
    if kind == "rrqr":
        n = size(8, 160)
        return {"kind": kind, "limbs": N, "m": n + size(8, 500), "n": n, "rhs": size(1, 16)}
    if kind == "mixed_lu":
        return {"kind": kind, "limbs": N, "n": size(200, 4096), "rhs": size(1, 32),
                "decades": rng.randint(3, 12)}
    if kind == "spd_batch":
        least = size(4, 40)
        return {"kind": kind, "limbs": N, "blocks": size(100, 10000 // 4 ** (N - 2)),
                "least": least, "most": size(least + 1, 256)}
    # one factorization and its solves: the wider types take longer at the same size
    return {"kind": kind, "limbs": N, "n": size(48, {2: 2000, 3: 1300, 4: 1000}[N]),
            "rhs": size(1, 64)}


# ----------------------------------------- multi-limb values in plain torch ----
def _two_sum(a, b):
    s = a + b
    t = s - a
    return s, (a - (s - t)) + (b - t)


def _accumulate(acc, p):
    """acc (a list, largest first) plus the float64 tensor p."""
    for i in range(len(acc)):
        acc[i], p = _two_sum(acc[i], p)
    return acc


def _limbs(acc, N):
    """The N leading limbs of the list's sum, each rounded to nearest of what remains."""
    x = list(acc)
    for _ in range(len(x) + 1):
        for i in range(len(x) - 1, 0, -1):
            x[i - 1], x[i] = _two_sum(x[i - 1], x[i])
    return x[:N]


def _plus(x, y, N):
    acc = [t.clone() for t in x] + [torch.zeros_like(x[0])] * (N + 1 - len(x))
    for t in y:
        _accumulate(acc, t)
    return _limbs(acc, N)


def _minus(x, y, N):
    return _plus(x, [-t for t in y], N)


def _slices(x, dim, bits, count):
    """Short slices whose sum is the multi-limb matrix down to 2^-(bits*count) of the largest
    entry of each row (dim -1) or column (dim -2); a row's slice is integers of at most
    `bits` bits times one power of two."""
    top = x[0].abs().amax(dim=dim, keepdim=True)
    e = torch.frexp(torch.where(top > 0, top, torch.ones_like(top)))[1].to(torch.float64)
    r, out = [t.clone() for t in x], []
    for s in range(1, count + 1):
        c = torch.ldexp(torch.ones_like(e), e + (52 - bits * s)) * 1.5
        q = torch.zeros_like(r[0])
        for i in range(len(r)):
            part = (r[i] + c) - c
            r[i] = r[i] - part
            q = q + part
        out.append(q)
    return out


def _slicing(k, N):
    bits = min(24, (51 - math.ceil(math.log2(max(k, 2)))) // 2)
    return bits, math.ceil((53 * N + 14) / bits)


def _mm(A, B, N):
    """A @ B (lists of limbs, or slices made before with _slices) to N limbs."""
    k = B[0].shape[-2]
    bits, count = _slicing(k, N)
    SA = A if isinstance(A, tuple) else _slices(A, -1, bits, count)
    SB = _slices(B, -2, bits, count)
    acc = None
    for level in range(count - 1, -1, -1):
        for i in range(level + 1):
            p = SA[i] @ SB[level - i]
            acc = [torch.zeros_like(p) for _ in range(N + 1)] if acc is None else acc
            _accumulate(acc, p)
    return _limbs(acc, N)


def _solve(A, B, N, symmetric=False):
    """A \\ B by refinement of a 64-bit factor, to N limbs."""
    bits, count = _slicing(A[0].shape[-1], N)
    SA = tuple(_slices(A, -1, bits, count))
    if symmetric:
        f = torch.linalg.cholesky(A[0])
        step = lambda r: torch.cholesky_solve(r, f)  # noqa: E731
    else:
        f, p = torch.linalg.lu_factor(A[0])
        step = lambda r: torch.linalg.lu_solve(f, p, r)  # noqa: E731
    X = [torch.zeros_like(B[0]) for _ in range(N)]
    R = B
    for _ in range(60):
        d = step(R[0])
        X = _plus(X, [d], N)
        if float(d.abs().max()) <= 2.0 ** -(53 * N + 4) * float(X[0].abs().max()):
            break
        R = _minus(B, _mm(SA, X, N), N)
    return X


def _chol(S, N):
    """The lower Cholesky factor to N limbs: first-order corrections of the 64-bit factor."""
    L0 = torch.linalg.cholesky(S[0])
    L = [L0] + [torch.zeros_like(L0)] * (N - 1)
    for _ in range(N + 2):
        E = _minus(S, _mm(L, [t.mT.contiguous() for t in L], N), N)[0]
        E = torch.linalg.solve_triangular(L0, E, upper=False)
        E = torch.linalg.solve_triangular(L0, E.mT.contiguous(), upper=False)
        E = torch.tril(E)
        E.diagonal().mul_(0.5)
        L = _plus(L, [L0 @ E], N)
    return L


def _lu(A, N):
    """The packed unit-lower / upper factor to N limbs and the 1-based row exchanges."""
    f, piv = torch.linalg.lu_factor(A[0])
    rows = list(range(A[0].shape[0]))
    for i, p in enumerate((piv - 1).tolist()):
        rows[i], rows[p] = rows[p], rows[i]
    PA = [t[rows] for t in A]
    eye = torch.eye(len(rows), dtype=torch.float64, device=f.device)
    L0, U0 = torch.tril(f, -1) + eye, torch.triu(f)
    zero = torch.zeros_like(f)
    L, U = [L0] + [zero] * (N - 1), [U0] + [zero] * (N - 1)
    for _ in range(N + 3):
        E = _minus(PA, _mm(L, U, N), N)[0]
        E = torch.linalg.solve_triangular(L0, E, upper=False, unitriangular=True)
        E = torch.linalg.solve_triangular(U0, E, upper=True, left=False)
        L = _plus(L, [L0 @ torch.tril(E, -1)], N)
        U = _plus(U, [torch.triu(E) @ U0], N)
    return [torch.tril(a, -1) + torch.triu(b) for a, b in zip(L, U)], piv


# ----------------------------------------------------------------- inputs ----
def _generator(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed))


def _randn(g, N, *shape, spread=0.0):
    """Normally distributed values (times 2^U(-spread, spread)) with every limb populated."""
    x = [torch.randn(shape, dtype=torch.float64, device="cuda", generator=g)]
    if spread:
        u = torch.rand(shape, dtype=torch.float64, device="cuda", generator=g)
        x[0] = x[0] * torch.exp2((2 * u - 1) * spread)
    for _ in range(N - 1):
        r = torch.randn(shape, dtype=torch.float64, device="cuda", generator=g)
        x.append(r * x[-1].abs() * 2.0 ** -53)
    return _limbs(x, N)


def _spd(g, N, n, *batch):
    """R R^T + n I, exactly symmetric."""
    R = _randn(g, N, *batch, n, n)
    S = _mm(R, [t.mT.contiguous() for t in R], N)
    S = [torch.tril(t) + torch.tril(t, -1).mT for t in S]
    shift = n * torch.eye(n, dtype=torch.float64, device="cuda").expand_as(S[0])
    return _plus(S, [shift], N)


def _classes(case, seed):
    """The batch's sizes (the same for every seed) and, for each size, the numbers of its blocks
    and their (S, b, w)."""
    sizes = np.random.RandomState(case["blocks"]).randint(case["least"], case["most"] + 1,
                                                          case["blocks"])
    g = _generator(seed)
    for s in np.unique(sizes):
        at = np.flatnonzero(sizes == s)
        s = int(s)
        yield sizes, at, (_spd(g, case["limbs"], s, len(at)),
                          _randn(g, case["limbs"], len(at), s, 1),
                          _randn(g, case["limbs"], len(at), s, 1))


def _inputs(case, seed):
    """The operands of every kind but the batch, as lists of limbs."""
    g, N, kind = _generator(seed), case["limbs"], case["kind"]
    if kind in ("gemm", "int8"):
        m, k, n = case["m"], case["k"], case["n"]
        spread = 20.0 if kind == "int8" else 0.0
        got = [_randn(g, N, m, k, spread=spread), _randn(g, N, k, n, spread=spread)]
        return got + ([_randn(g, N, m, n)] if case.get("update") else [])
    if kind == "gemv":
        m, n = case["m"], case["n"]
        return [_randn(g, N, m, n), _randn(g, N, n if case["trans"] == "N" else m, 1)]
    if kind == "rrqr":
        return [_randn(g, N, case["m"], case["n"]), _randn(g, N, case["m"], case["rhs"])]
    n = case["n"]
    if kind == "chol":
        A = _spd(g, N, n)
    elif kind == "lu":
        A = _randn(g, N, n, n)
    elif kind == "ldlt":  # a saddle-point matrix: [H G^T; G 0], H indefinite
        A = _randn(g, N, n, n)
        A = [torch.tril(t) + torch.tril(t, -1).mT for t in A]
        c = n - n // 4
        for t in A:
            t[c:, c:] = 0.0
    else:  # mixed_lu: U diag(sigma) V^T with singular values from 1 to 10^-decades
        U, V = (torch.linalg.qr(torch.randn((n, n), dtype=torch.float64, device="cuda",
                                            generator=g))[0] for _ in range(2))
        sigma = torch.logspace(0.0, -float(case["decades"]), n, dtype=torch.float64,
                               device="cuda")
        W = sigma[:, None] * V.mT
        A = _mm([U], [W], N)
    return [A, _randn(g, N, n, case["rhs"])]


def _planes(x):
    """Limb planes of a matrix as the library stores them: (N, columns, rows)."""
    return torch.stack([t.mT for t in x]).contiguous()


def prepare(case, seed):
    mf = _package()
    kind, N = case["kind"], case["limbs"]
    if kind == "spd_batch":
        batch = S0 = B0 = W = None
        for sizes, at, (S, b, w) in _classes(case, seed):
            if batch is None:
                batch = mf.batched.SPDBatch(N, sizes)
                S0, B0 = torch.zeros_like(batch.S), torch.zeros_like(batch.X)
                W = torch.zeros_like(batch.X)
            s = S[0].shape[-1]
            o = torch.as_tensor(batch.offsets_host[at], device="cuda")[:, None]
            v = torch.as_tensor(batch.boffsets_host[at], device="cuda")[:, None]
            o = o + torch.arange(s * s, device="cuda")
            v = v + torch.arange(s, device="cuda")
            for l in range(N):
                S0[l, o] = S[l].reshape(len(at), s * s)
                B0[l, v] = b[l][:, :, 0]
                W[l, v] = w[l][:, :, 0]
        return {"case": case, "batch": batch, "S": S0, "b": B0, "w": W}
    ops = [mf.MFMatrix.from_tensor(_planes(x)) for x in _inputs(case, seed)]
    if kind == "gemv":
        m, n = (case["m"], case["n"]) if case["trans"] == "N" else (case["n"], case["m"])
        x = mf.MFMatrix.from_tensor(ops[1].storage, is_vector=True)
        return {"case": case, "ops": [ops[0], x], "out": mf.MFMatrix.zeros(N, m)}
    state = {"case": case, "ops": ops}
    if kind in ("gemm", "int8"):
        state["out"] = mf.MFMatrix.zeros(N, case["m"], case["n"])
    return state


# -------------------------------------------------------------------- run ----
def run(state):
    mf = _package()
    case = state["case"]
    kind = case["kind"]
    if kind == "spd_batch":
        batch = state["batch"]
        batch.S.copy_(state["S"])
        batch.X.copy_(state["b"])
        x, pullback = mf.batched.solve_spd_batched_rrule(batch)
        Sbar, bbar = pullback(state["w"])
        return {"x": x, "Sbar": Sbar, "bbar": bbar}
    A, B = state["ops"][:2]
    if kind == "gemm":
        C = state["out"]
        if case["update"]:
            C.copy_(state["ops"][2])
            return [mf.gemm_(C, A, B, -1.0, 1.0).storage]
        return [mf.gemm_(C, A, B).storage]
    if kind == "int8":
        config = mf.KernelConfig(gemm_strategy="ozaki", ozaki_scheme="modular")
        return [mf.gemm_(state["out"], A, B, config=config).storage]
    if kind == "gemv":
        return [mf.gemv_(state["out"], A, B, trans=case["trans"]).storage]
    if kind == "mixed_lu":
        X, _ = mf.solve_mixed_lu(A, B)
        return {"X": X.storage}
    if kind == "rrqr":
        F = mf.rrqr_(A.copy())
        rank = mf.numerical_rank(F, rtol=1e-12)
        Y = mf.apply_q_(B.copy(), F, "T")
        Z = Y.view(slice(0, rank))
        mf.solve_r_(Z, F, rank)
        return {"X": Z.planes(), "factors": F.factors.storage, "tau": F.tau,
                "permutation": F.permutation, "rank": rank}
    factor = {"chol": mf.cholesky_, "lu": mf.lu_, "ldlt": mf.ldlt_}[kind]
    F = factor(A.copy())
    X = mf.solve(F, B)
    out = {"X": X.storage, "factors": F.factors.storage}
    if kind == "lu":
        out["pivots"] = F.ipiv
    if kind == "ldlt":
        out.update(subdiagonal=F.dsub, pivots=F.pivots, blocks=F.blocks)
    return out


# ------------------------------------------------------------------- work ----
#: binary64 operations of one multi-double multiply-add, by limbs
MAC = {2: 28.0, 3: 99.0, 4: 227.0}


def work(case):
    """Inputs read once and results written once; binary64 operations of the multi-double
    steps, and for the tensor-core products the 8-bit operations of the residues."""
    N, kind = case["limbs"], case["kind"]
    value, mac = 8.0 * N, MAC[case["limbs"]]
    if kind in ("gemm", "int8"):
        m, k, n = case["m"], case["k"], case["n"]
        values = m * k + k * n + m * n * (2 if case.get("update") else 1)
        terms = (2 * 53 * N + 28) // 8 * 2.0 if kind == "int8" else mac
        return {"bytes": value * values, "flops": terms * m * n * k}
    if kind == "gemv":
        m, n = case["m"], case["n"]
        return {"bytes": value * (m * n + m + n), "flops": mac * m * n}
    if kind == "rrqr":
        m, n, r = case["m"], case["n"], case["rhs"]
        return {"bytes": value * (2 * m * n + m * r + n * r),
                "flops": mac * (m * n * n - n ** 3 / 3 + 2 * m * n * r)}
    if kind == "spd_batch":
        s = np.arange(case["least"], case["most"] + 1, dtype=np.float64)
        one, two, three = (case["blocks"] * float(np.mean(s ** p)) for p in (1, 2, 3))
        return {"bytes": value * (2.5 * two + 4 * one),
                "flops": mac * (three / 6 + 2 * two + two)}
    n, r = case["n"], case["rhs"]
    if kind == "mixed_lu":  # the binary64 factor and one residual of full precision
        return {"bytes": value * (n * n + 2 * n * r), "flops": 2 * n ** 3 / 3 + mac * n * n * r}
    share = {"chol": 1 / 6, "lu": 1 / 3, "ldlt": 1 / 6}[kind]
    half = 1.0 if kind == "lu" else 0.5
    return {"bytes": value * (2 * half * n * n + 2 * n * r),
            "flops": mac * (share * n ** 3 + n * n * r)}


# ------------------------------------------------------------------ exact ----
def exact(case, seed):
    N, kind = case["limbs"], case["kind"]
    if kind == "spd_batch":
        out = None
        for sizes, at, (S, b, w) in _classes(case, seed):
            if out is None:
                sq, length = sizes.astype(np.int64) ** 2, sizes.astype(np.int64)
                so, vo = np.cumsum(sq) - sq, np.cumsum(length) - length
                empty = lambda t: torch.zeros((N, int(t)), dtype=torch.float64,  # noqa: E731
                                              device="cuda")
                out = {"x": empty(length.sum()), "Sbar": empty(sq.sum()),
                       "bbar": empty(length.sum())}
            s = S[0].shape[-1]
            o = torch.as_tensor(so[at], device="cuda")[:, None]
            v = torch.as_tensor(vo[at], device="cuda")[:, None]
            o, v = o + torch.arange(s * s, device="cuda"), v + torch.arange(s, device="cuda")
            both = _solve(S, [torch.cat([p, q], -1) for p, q in zip(b, w)], N, symmetric=True)
            x, y = [t[..., :1] for t in both], [t[..., 1:] for t in both]
            half = [-0.5 * t for t in _mm(y, [t.mT.contiguous() for t in x], N)]
            G = _plus(half, [t.mT for t in half], N)
            for l in range(N):
                out["x"][l, v], out["bbar"][l, v] = x[l][:, :, 0], y[l][:, :, 0]
                out["Sbar"][l, o] = G[l].reshape(len(at), s * s)
        return out
    ops = _inputs(case, seed)
    A, B = ops[:2]
    if kind in ("gemm", "int8"):
        P = _mm(A, B, N)
        return [_planes(_minus(ops[2], P, N) if case.get("update") else P)]
    if kind == "gemv":
        return [_planes(_mm(A if case["trans"] == "N" else [t.mT.contiguous() for t in A], B, N))]
    if kind == "rrqr":  # [I A; A^T 0] [r; x] = [b; 0]: the least-squares solution, as pivoted
        m, n = case["m"], case["n"]
        K = [torch.zeros((m + n, m + n), dtype=torch.float64, device="cuda") for _ in range(N)]
        for t, a in zip(K, A):
            t[:m, m:], t[m:, :m] = a, a.mT
        K[0].diagonal()[:m] = 1.0
        rhs = [torch.cat([t, t.new_zeros(n, t.shape[1])]) for t in B]
        X = [t[m:] for t in _solve(K, rhs, N)]
        left, order = A[0].clone(), []
        for _ in range(n):  # the pivot order: the column with the most left
            j = int(torch.argmax((left * left).sum(0)))
            order.append(j)
            q = left[:, j] / left[:, j].norm()
            left = left - torch.outer(q, q @ left)
            left[:, order] = 0.0
        return {"X": _planes([t[order] for t in X])}
    out = {"X": _planes(_solve(A, B, N))}
    if kind == "chol":
        L = _chol(A, N)
        out["factors"] = _planes([torch.tril(t) + torch.triu(a, 1) for t, a in zip(L, A)])
    if kind == "lu":
        out["factors"] = _planes(_lu(A, N)[0])
    return out
