"""Workloads whose time is tracked: what a program has this library do, through its public entry
points, over the sizes it meets.

Kinds of case:

* ``solve``       a kept solver handle takes new data vectors (``update``) and solves to the
                  default gap of 1e-8: the parameter sweep of a conic program.
* ``iteration``   one interior-point iteration of a host that keeps its own driver and calls the
                  kernel-level entry points: NT scaling, Schur assembly, factorisation, a refined
                  KKT solve of two right-hand sides, step length.
* ``split_dgemm`` a binary64 matrix product on the INT8 tensor cores, device buffers.
* ``rns_gemm``    an exact MpFloat matrix product, rounded once, on host or on device buffers.
* ``rns_congruence`` the exact congruence A X A' behind the MPFR PSD transforms, host buffers.
* ``mp_ldl``      the dense MPFR LDL' of a Schur complement in device memory, in place.
* ``mp_cone``     the MPFR cone work of an iteration: NT scaling of PSD blocks and the step-length
                  bounds of both directions.

A drawn ``solve`` is of the dense family; the rank-one family is drawn as ``iteration``.

Families of a ``solve`` or ``iteration``: ``dense`` (one PSD block of order n, m dense symmetric
constraints) and ``rank1`` (the bootstrap shape: PSD blocks whose orders spread evenly over
nmin..nmax, every constraint four rank-one terms of their Chebyshev bases).
"""
import math
import os
import sys

import numpy as np
import torch

_ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
sys.path.insert(0, os.path.join(_ROOT, "sdpx.rs_b200"))

from sdpx_b200 import _lib, problems  # noqa: E402
from sdpx_b200.solver import DefaultSettings, DefaultSolver, KernelContext  # noqa: E402

C = _lib.C
TOUCH = 4  # blocks a rank-one constraint touches


def _tri(n):
    return n * (n + 1) // 2


def listed():
    return [
        # the smallest call: a projection-sized SDP, bound by launches and host round trips
        {"name": "solve_small", "kind": "solve", "family": "dense", "n": 16, "m": 40},
        # the plain dense SDP
        {"name": "solve_dense", "kind": "solve", "family": "dense", "n": 50, "m": 200},
        # the bootstrap-shaped SDP, whole
        {"name": "solve_bootstrap", "kind": "solve", "family": "rank1", "blocks": 32, "m": 2000,
         "nmin": 10, "nmax": 60},
        # one iteration of a foreign driver on the dense SDP (dense constraint columns)
        {"name": "iteration_dense", "kind": "iteration", "family": "dense", "n": 50, "m": 200, "split": False},
        # one iteration on the bootstrap shape, the factorisation's products in split precision
        {"name": "iteration_split", "kind": "iteration", "family": "rank1", "blocks": 32, "m": 2000,
         "nmin": 10, "nmax": 60, "split": True},
        # one iteration of the precision workload, plain FP64 factorisation
        {"name": "iteration_precision", "kind": "iteration", "family": "rank1", "blocks": 64, "m": 4000,
         "nmin": 10, "nmax": 60, "split": False},
        # a trailing update of a large factorisation
        {"name": "split_dgemm_2048", "kind": "split_dgemm", "m": 2048, "n": 2048, "k": 2048,
         "ta": "N", "tb": "N"},
        # one exact product of block-sized matrices at 512 bits, host to host
        {"name": "rns_gemm_63", "kind": "rns_gemm", "limbs": 8, "m": 63, "n": 63, "k": 63, "ta": "N",
         "tb": "N", "upper": False, "device": False},
        # a trailing update of the 256-bit factorisation, resident
        {"name": "rns_gemm_2000", "kind": "rns_gemm", "limbs": 4, "m": 2000, "n": 2000, "k": 2000,
         "ta": "N", "tb": "T", "upper": False, "device": True},
        # a PSD block's congruence at 256 bits
        {"name": "rns_congruence_60", "kind": "rns_congruence", "limbs": 4, "m": 60, "k": 60},
        # the 256-bit Schur complement's factorisation
        {"name": "mp_ldl_1000", "kind": "mp_ldl", "limbs": 4, "n": 1000},
        # the 256-bit cone work of eight PSD blocks
        {"name": "mp_cone_256", "kind": "mp_cone", "limbs": 4, "blocks": 8, "nmin": 10, "nmax": 40},
    ]


def _log_int(rng, lo, hi):
    """An integer spread over the logarithm of lo..hi."""
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["solve", "solve", "iteration", "iteration", "split_dgemm", "rns_gemm", "rns_gemm",
                       "rns_congruence", "mp_ldl", "mp_cone"])
    if kind in ("solve", "iteration"):
        if kind == "solve" or rng.random() < 0.5:
            n = rng.randint(12, 64)
            case = {"kind": kind, "family": "dense", "n": n, "m": rng.randint(20, min(300, n * (n + 1) // 3))}
        else:
            case = {"kind": kind, "family": "rank1", "blocks": _log_int(rng, 6, 63), "nmin": 10, "nmax": 60}
            # the v v' of a block span 2n - 1 dimensions: fewer constraints than that in all, so
            # that the Schur complement is regular
            span = sum(2 * n - 1 for n in _orders(case))
            case["m"] = int(span * rng.uniform(0.6, 0.915))
        if kind == "iteration":
            case["split"] = case["m"] >= 1024 and rng.random() < 0.5
        return case
    if kind == "split_dgemm":
        return {"kind": kind, "m": _log_int(rng, 200, 2048), "n": _log_int(rng, 200, 2048),
                "k": _log_int(rng, 200, 2048), "ta": rng.choice("NT"), "tb": rng.choice("NT")}
    if kind == "rns_gemm":
        device = rng.random() < 0.6
        top = 1800 if device else 160
        return {"kind": kind, "limbs": rng.choice([2, 3, 4]) if device else rng.choice([2, 4, 6, 8]),
                "m": _log_int(rng, 24, top), "n": _log_int(rng, 24, top), "k": _log_int(rng, 24, top),
                "ta": rng.choice("NT"), "tb": rng.choice("NT"), "upper": rng.random() < 0.3, "device": device}
    if kind == "rns_congruence":
        return {"kind": kind, "limbs": rng.choice([2, 4, 6]), "m": rng.randint(10, 64), "k": rng.randint(10, 64)}
    if kind == "mp_ldl":
        limbs = rng.choice([2, 4, 4, 8])
        return {"kind": kind, "limbs": limbs, "n": _log_int(rng, 40, 1000 if limbs <= 4 else 400)}
    return {"kind": kind, "limbs": rng.choice([2, 4]), "blocks": rng.randint(1, 8), "nmin": rng.randint(4, 12),
            "nmax": rng.randint(14, 40)}


# ---- MpFloat elements: limbs u64 (least significant first), i32 kind (sign x 3), i32 exponent ----


def _mp(x, limbs, rng):
    """MpFloat<limbs> elements with the leading bits of the non-zero binary64 x and random bits
    below them: uint8 array of shape x.shape + (8 * limbs + 8,)."""
    x = np.asarray(x, dtype=np.float64)
    frac, ex = np.frexp(np.abs(x))
    el = np.zeros(x.shape, dtype=[("limb", "<u8", (limbs,)), ("kind", "<i4"), ("exp", "<i4")])
    el["limb"] = rng.integers(0, 1 << 64, size=x.shape + (limbs,), dtype=np.uint64)
    top = np.ldexp(frac, 53).astype(np.uint64) << np.uint64(11)
    el["limb"][..., limbs - 1] = top | (el["limb"][..., limbs - 1] >> np.uint64(53))
    el["kind"] = np.where(x < 0, -3, 3)
    el["exp"] = ex
    return el.view(np.uint8).reshape(x.shape + (8 * limbs + 8,))


def _mp_matrix(X, limbs, rng):
    """Column-major MpFloat bytes of a matrix."""
    return np.ascontiguousarray(_mp(np.asarray(X).T, limbs, rng))


def _mp_symmetric(X, limbs, rng):
    """Column-major MpFloat bytes of a matrix, exactly symmetric."""
    el = _mp_matrix(X, limbs, rng)
    i, j = np.tril_indices(X.shape[0], -1)
    el[i, j] = el[j, i]
    return el


def _wide(rng, *shape):
    """Entries of either sign spread over a few orders of magnitude."""
    return rng.standard_normal(shape) * np.exp2(rng.uniform(-12.0, 12.0, size=shape))


# ---- interior points ----


def _interior(orders, rng):
    """Blocks (S, Z) of an iterate near the central path: S of spread eigenvalues, S Z close to
    mu I without commuting."""
    out = []
    for n in orders:
        Q = np.linalg.qr(rng.standard_normal((n, n)))[0]
        w = 10.0 ** rng.uniform(-1.0, 1.0, n)
        S = (Q * w) @ Q.T
        E = rng.standard_normal((n, n)) / math.sqrt(n)
        L = Q * np.sqrt(w)
        K = np.linalg.inv(L).T
        Z = 0.1 * (K @ (np.eye(n) + 0.15 * (E + E.T) / math.sqrt(2.0)) @ K.T)
        out.append((0.5 * (S + S.T), 0.5 * (Z + Z.T)))
    return out


def _svecs(mats):
    return np.concatenate([problems.svec(M) for M in mats])


def _direction(orders, rng):
    return _svecs([E + E.T for E in (rng.standard_normal((n, n)) for n in orders)])


def _orders(case):
    """Block orders spread evenly over nmin..nmax."""
    b, lo, hi = case["blocks"], case["nmin"], case["nmax"]
    return [lo + (k * 7919 % b) * (hi - lo) // max(b - 1, 1) for k in range(b)]


def _basis(n):
    """Chebyshev polynomials 0..n-1 at 2n nodes: n x 2n."""
    t = (2 * np.arange(2 * n) + 1) * np.pi / (4 * n)
    return np.cos(np.outer(np.arange(n), t))


def _rank1_problem(case, seed):
    """min -b'y s.t. C - sum_i y_i A_i >= 0 per block, A_i four terms w v v' on four blocks:
    strictly feasible on both sides (X = I, C = sum_i y0_i A_i + I)."""
    rng = np.random.default_rng(seed)
    orders, m = _orders(case), case["m"]
    nb = len(orders)
    ns = np.array(orders)
    blk = np.sort(np.argsort(rng.random((m, nb)), axis=1)[:, :TOUCH], axis=1)
    col = (rng.random((m, TOUCH)) * 2 * ns[blk]).astype(np.int64)
    wgt = rng.uniform(0.5, 2.0, size=(m, TOUCH))
    y0 = rng.standard_normal(m)
    cols = []  # svec(v v') of every basis column of every block
    bcon, bprim, size, offs = [], np.zeros(m), _tri(ns), np.concatenate([[0], np.cumsum(_tri(ns))])
    for j, n in enumerate(orders):
        V = _basis(n)
        i, jj = problems.svec_index(n)
        cols.append(np.where(i == jj, 1.0, problems.SQRT2)[None, :] * (V[i] * V[jj]).T)
        at, slot = np.nonzero(blk == j)
        np.add.at(bprim, at, wgt[at, slot] * np.sum(V * V, axis=0)[col[at, slot]])
        d = np.bincount(col[at, slot], weights=y0[at] * wgt[at, slot], minlength=2 * n)
        bcon.append(problems.svec((V * d) @ V.T + np.eye(n)))
    count = size[blk].sum(axis=1)
    indptr = np.concatenate([[0], np.cumsum(count)])
    vals, rows = np.empty(indptr[-1]), np.empty(indptr[-1], dtype=np.int64)
    p = 0
    for c in range(m):
        for j, k, w in zip(blk[c], col[c], wgt[c]):
            q = p + size[j]
            np.multiply(cols[j][k], w, out=vals[p:q])
            rows[p:q] = np.arange(offs[j], offs[j + 1])
            p = q
    A = problems.sp.csc_matrix((vals, rows, indptr), shape=(int(offs[-1]), m))
    return problems.ConicProblem(P=None, q=-bprim, A=A, b=np.concatenate(bcon),
                                 cones=[("psd", n) for n in orders])


def _problem(case, seed):
    if case["family"] == "dense":
        return problems.dense_sdp(case["n"], case["m"], seed=seed)
    return _rank1_problem(case, seed)


def _iteration_inputs(case, seed):
    prob = _problem(case, seed)
    rng = np.random.default_rng(seed + 1)
    orders = [d for _, d in prob.cones]
    pts = _interior(orders, rng)
    return {"prob": prob, "orders": orders, "s": _svecs([p[0] for p in pts]), "z": _svecs([p[1] for p in pts]),
            "bx": rng.standard_normal((2, prob.n)), "bz": rng.standard_normal((2, prob.m)),
            "dz": _direction(orders, rng), "ds": _direction(orders, rng)}


def _cone_inputs(case, seed):
    rng = np.random.default_rng(seed)
    limbs = case["limbs"]
    orders = _orders(case)
    pts = _interior(orders, rng)

    def mp(v):
        return _mp(v, limbs, rng).tobytes()

    return {"orders": orders, "s": mp(_svecs([p[0] for p in pts])), "z": mp(_svecs([p[1] for p in pts])),
            "ds": mp(_direction(orders, rng)), "dz": mp(_direction(orders, rng)),
            "one": _mp_power(0, limbs)}


def _mp_power(e, limbs):
    """2^e as one MpFloat."""
    el = np.zeros(1, dtype=[("limb", "<u8", (limbs,)), ("kind", "<i4"), ("exp", "<i4")])
    el["limb"][0, limbs - 1] = 1 << 63
    el["kind"], el["exp"] = 3, e + 1
    return el.tobytes()


def prepare(case, seed):
    kind = case["kind"]
    st = {"case": case}
    if kind == "solve":
        prob = _problem(case, seed)
        st["solver"] = DefaultSolver(prob.P, prob.q, prob.A, prob.b, prob.cones,
                                     DefaultSettings(kkt_form="condensed"))
        st["q"], st["b"] = prob.q, prob.b
        return st
    if kind == "iteration":
        st.update(_iteration_inputs(case, seed))
        st["ctx"] = KernelContext()
        st["ctx"].upload(st["prob"].A, st["orders"])
        st["ctx"].set_factor_form(1 if case["split"] else 0)
        return st
    if kind == "mp_cone":
        st.update(_cone_inputs(case, seed))
        st["ctx"] = KernelContext()
        return st
    st["ctx"] = KernelContext()
    rng = np.random.default_rng(seed)
    if kind == "split_dgemm":
        A, B = _dgemm_inputs(case, seed)
        st["A"], st["B"] = A.cuda(), B.cuda()  # column-major: rows of these tensors are columns
        st["out"] = torch.empty((case["n"], case["m"]), dtype=torch.float64, device="cuda")
    elif kind == "rns_gemm":
        L, m, n, k = case["limbs"], case["m"], case["n"], case["k"]
        A = _mp_matrix(_wide(rng, *((m, k) if case["ta"] == "N" else (k, m))), L, rng)
        B = _mp_matrix(_wide(rng, *((k, n) if case["tb"] == "N" else (n, k))), L, rng)
        if case["device"]:
            st["A"], st["B"] = torch.from_numpy(A).cuda(), torch.from_numpy(B).cuda()
            st["out"] = torch.empty((n, m, 8 * L + 8), dtype=torch.uint8, device="cuda")
        else:
            st["A"], st["B"] = A.tobytes(), B.tobytes()
    elif kind == "rns_congruence":
        L, m, k = case["limbs"], case["m"], case["k"]
        st["A"] = _mp_matrix(_wide(rng, m, k), L, rng).tobytes()
        X = rng.standard_normal((k, k))
        st["X"] = _mp_symmetric(X + X.T, L, rng).tobytes()
    else:  # mp_ldl: a Schur complement, positive definite with a graded diagonal
        n, L = case["n"], case["limbs"]
        G = rng.standard_normal((n, n + 8))
        g = np.exp2(rng.uniform(-4.0, 4.0, n))
        st["A"] = torch.from_numpy(_mp_symmetric((G @ G.T / n + np.eye(n)) * np.outer(g, g), L, rng)).cuda()
        st["F"] = torch.empty_like(st["A"])
        st["D"] = torch.empty((n, 8 * L + 8), dtype=torch.uint8, device="cuda")
    torch.cuda.synchronize()
    return st


def _dgemm_inputs(case, seed):
    g = torch.Generator().manual_seed(seed)
    ar = (case["k"], case["m"]) if case["ta"] == "N" else (case["m"], case["k"])
    br = (case["n"], case["k"]) if case["tb"] == "N" else (case["k"], case["n"])
    return (torch.randn(ar, dtype=torch.float64, generator=g), torch.randn(br, dtype=torch.float64, generator=g))


def run(st):
    case = st["case"]
    kind = case["kind"]
    if kind == "solve":
        st["solver"].update(st["q"], st["b"])
        sol = st["solver"].solve()
        out = {"x": sol.x, "s": sol.s, "primal": sol.obj_val, "dual": sol.obj_val_dual,
               "status": int(sol.status_code), "iterations": int(sol.iterations)}
        # a bootstrap program reads the functional x and its slack s; the multipliers of the rank-one
        # family are nearly degenerate, and a gap of 1e-8 leaves them free in the ninth digit
        # (measured: data moved by one rounding move z by up to 1e-9, and x and s by 1e-11)
        if case["family"] == "dense":
            out["z"] = sol.z
        return out
    ctx = st["ctx"]
    if kind == "iteration":
        lam, _ = ctx.nt_scale(st["s"], st["z"])
        _lib.call("sdpxg_schur_assemble", ctx._h, None)
        bad = ctx.factor(1e-8)
        sols = [ctx.kkt_solve(bx, bz) for bx, bz in zip(st["bx"], st["bz"])]
        alpha, _ = ctx.step_length(st["dz"], st["ds"], 1.0)
        return {"lam": lam, "x": [s[0] for s in sols], "z": [s[1] for s in sols], "alpha": float(alpha),
                "failed": int(bad)}
    if kind == "split_dgemm":
        A, B, out = st["A"], st["B"], st["out"]
        ctx.split_dgemm_device(case["ta"], case["tb"], case["m"], case["n"], case["k"], 1.0, A.data_ptr(),
                               A.shape[1], B.data_ptr(), B.shape[1], 0.0, out.data_ptr(), case["m"])
        return out
    if kind == "rns_gemm":
        A, B = st["A"], st["B"]
        m, n, k = case["m"], case["n"], case["k"]
        lda, ldb = (m if case["ta"] == "N" else k), (k if case["tb"] == "N" else n)
        if case["device"]:
            ctx.rns_gemm_device(case["limbs"], case["ta"], case["tb"], m, n, k, A.data_ptr(), lda,
                                B.data_ptr(), ldb, st["out"].data_ptr(), case["upper"])
            return st["out"]
        raw, _ = ctx.rns_gemm(case["limbs"], case["ta"], case["tb"], m, n, k, A, lda, B, ldb, case["upper"])
        return np.frombuffer(raw, dtype=np.uint8)
    if kind == "rns_congruence":
        raw, _ = ctx.rns_congruence(case["limbs"], "N", case["m"], case["k"], st["A"], case["m"], st["X"],
                                    case["k"])
        return np.frombuffer(raw, dtype=np.uint8)
    if kind == "mp_ldl":
        F, D, n = st["F"], st["D"], case["n"]
        F.copy_(st["A"])  # the factorisation works in place
        torch.cuda.current_stream().synchronize()  # its operands have to be complete
        bad = C.c_uint32()
        _lib.call("sdpxg_mp_ldl_device", ctx._h, case["limbs"], n, C.c_void_p(F.data_ptr()), n, None,
                  C.c_void_p(D.data_ptr()), C.byref(bad))
        return {"L": F, "dinv": D, "failed": int(bad.value)}
    limbs, orders = case["limbs"], st["orders"]
    lam, lis, R, Ri, G, fail, _ = ctx.mp_nt_scale(limbs, orders, st["s"], st["z"])
    one = st["one"]
    ad, pd, _ = ctx.mp_step_length(limbs, orders, False, st["dz"], R, lis, one)
    ap, pp, _ = ctx.mp_step_length(limbs, orders, True, st["ds"], Ri, lis, one)
    raw = [np.frombuffer(v, dtype=np.uint8) for v in (lam, lis, R, Ri, G, ad, ap)]
    return {"raw": raw, "paths": np.array([fail, pd, pp], dtype=np.int64)}


def _rank1_sizes(case):
    """Mean order, mean triangle and columns per block of a rank-one family."""
    ns = _orders(case)
    n1 = sum(ns) / len(ns)
    tri = sum(_tri(n) for n in ns) / len(ns)
    n3 = sum(n ** 3 for n in ns) / len(ns)
    return n1, tri, n3, case["m"] * TOUCH / case["blocks"]


def work(case):
    kind = case["kind"]
    if kind in ("solve", "iteration"):
        m = case["m"]
        if case["family"] == "dense":
            n, tri, b = case["n"], _tri(case["n"]), 1
            data = 8.0 * tri * m
            schur = 4.0 * m * n ** 3 + 2.0 * m * m * tri
            cone = 60.0 * n ** 3
        else:
            n1, tri, n3, k = _rank1_sizes(case)
            b = case["blocks"]
            data = 8.0 * b * k * n1
            schur = b * (2.0 * k * n1 * n1 + k * k * n1)
            cone = 60.0 * b * n3
        step = schur + cone + m ** 3 / 3.0 + 8.0 * m * m
        iters = 12.0 if kind == "solve" else 1.0
        return {"bytes": data + 8.0 * (4.0 * b * tri + 4.0 * m) + 8.0 * m * m, "flops": iters * step}
    if kind == "split_dgemm":
        m, n, k = case["m"], case["n"], case["k"]
        return {"bytes": 8.0 * (m * k + k * n + m * n), "flops": 2.0 * m * n * k}
    L = case["limbs"]
    esz, words = 8.0 * L + 8.0, (2.0 * L) ** 2  # 32-bit word products of one full product
    if kind == "rns_gemm":
        m, n, k = case["m"], case["n"], case["k"]
        return {"bytes": esz * (m * k + k * n + m * n), "flops": 2.0 * m * n * k * words}
    if kind == "rns_congruence":
        m, k = case["m"], case["k"]
        return {"bytes": esz * (m * k + k * k + m * m), "flops": 2.0 * (k * k * m + k * m * m) * words}
    if kind == "mp_ldl":
        n = case["n"]
        return {"bytes": esz * (2.0 * n * n + n), "flops": n ** 3 / 3.0 * words}
    ns = _orders(case)
    n2, n3 = sum(n * n for n in ns) / len(ns), sum(n ** 3 for n in ns) / len(ns)
    return {"bytes": esz * case["blocks"] * 5.0 * n2, "flops": case["blocks"] * 60.0 * n3 * words}


def _exact_iteration(case, seed):
    st = _iteration_inputs(case, seed)
    prob = st["prob"]
    A = prob.A.tocsr()
    lams, blocks, row, alpha = [], [], 0, 1.0
    for n in st["orders"]:
        t = _tri(n)
        sl = slice(row, row + t)
        S, Z = problems.smat(st["s"][sl], n), problems.smat(st["z"][sl], n)
        L1, L2 = np.linalg.cholesky(S), np.linalg.cholesky(Z)
        U, lam, _ = np.linalg.svd(L2.T @ L1)
        r = np.sqrt(lam)
        R = np.linalg.solve(L2.T, U) * r
        Ri = (U.T @ L2.T) / r[:, None]
        lams.append(lam)
        blocks.append((sl, n, Ri.T @ Ri))
        for D in (R.T @ problems.smat(st["dz"][sl], n) @ R, Ri @ problems.smat(st["ds"][sl], n) @ Ri.T):
            lo = float(np.linalg.eigvalsh(D / np.outer(r, r))[0])
            if lo < 0:
                alpha = min(alpha, -1.0 / lo)
        row += t

    def hinv(v):
        return np.concatenate([problems.svec(G @ problems.smat(v[sl], n) @ G) for sl, n, G in blocks])

    H = np.zeros((prob.n, prob.n))
    for sl, n, G in blocks:
        Aj = A[sl].tocsc()
        cols = np.flatnonzero(np.diff(Aj.indptr))
        D = np.asarray(Aj[:, cols].todense())
        i, j = problems.svec_index(n)
        scale = np.where(i == j, 1.0, 1.0 / problems.SQRT2)[:, None]
        M = np.zeros((n, n, cols.size))
        M[i, j] = D * scale
        M[j, i] = D * scale
        T = np.einsum("ab,bck->ack", G, M, optimize=True)
        T = np.einsum("ack,cd->adk", T, G, optimize=True)
        H[np.ix_(cols, cols)] += D.T @ (T[i, j] / scale)
    xs, zs = [], []
    for bx, bz in zip(st["bx"], st["bz"]):
        rhs = bx + A.T @ hinv(bz)
        x = np.linalg.solve(H, rhs)
        x += np.linalg.solve(H, rhs - H @ x)
        xs.append(x)
        zs.append(hinv(A @ x - bz))
    return {"lam": np.concatenate(lams), "x": xs, "z": zs, "alpha": alpha, "failed": None}


def exact(case, seed):
    """Plain numpy of the cases that have a value: a whole solve stops at its gap, and MpFloat
    results are bytes."""
    if case["kind"] == "split_dgemm":
        A, B = (t.numpy() for t in _dgemm_inputs(case, seed))
        A = A.T if case["ta"] == "N" else A  # the tensors hold columns: op(A) is m x k
        B = B.T if case["tb"] == "N" else B
        return np.ascontiguousarray((A @ B).T)
    if case["kind"] == "iteration":
        return _exact_iteration(case, seed)
    return None
