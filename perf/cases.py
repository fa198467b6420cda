"""Workloads of the solver as its users run it: what each stands for, its inputs
(made on the GPU from a seed), one pass through the public entry points, the
bytes and operations a pass cannot do without, and its result in 64 bits.

Kinds
  solve        one system, device arrays: a controller's solve at every control step
  solve_host   one system, host arrays: the reference's solvePCG / pcg_solve call
  batch        a plan of many independent systems: sampling-based and multi-agent
               control, dataset generation, training
  batch_host   the same from pinned host memory, Phi^-1 built on the GPU
  pair         forward solve and adjoint of a loss: learning through the solver
  refine       ill-conditioned FP64 systems by FP32 PCG with FP64 refinement
  schur        S, gamma (and Phi^-1) from the problem data, before a solve
  backsub      states and controls from the multipliers, after a solve
  jacobi       the block-Jacobi Phi^-1 of a batch, at every new linearisation

Problems follow the workload generator of this repository: dynamics A_k with
N(0, 1/n) entries scaled to a spectral radius of 0.98 (here its estimate
||A^64||^(1/64), quick on the GPU), B_k ~ N(0, 1), Q = diag U[1, 10],
R = diag U[0.1, 1] (ill-conditioned: log-uniform), gamma ~ N(0, 1).
"""
import math
import os
import random
import sys

import numpy as np
import torch

_PKG = os.path.join(os.getcwd(), "gbd-pcg_gb300")
if _PKG not in sys.path:
    sys.path.insert(0, _PKG)
import gbdpcg  # noqa: E402

DEV = "cuda"


def listed():
    return [
        # the smallest: one short-horizon solve of a 14-state arm, as a controller makes it
        {"name": "solve n14 N32 f32", "kind": "solve", "n": 14, "N": 32, "f64": False, "tri": False},
        # a caller of the reference's host interface, with its block-tridiagonal layout for Phi^-1
        {"name": "solvePCG host n14 N128 f64", "kind": "solve_host", "n": 14, "N": 128, "f64": True, "tri": True},
        # one long horizon (trajectory smoothing): the rows are past what a cluster holds on chip
        {"name": "solve n14 N8192 f32", "kind": "solve", "n": 14, "N": 8192, "f64": False, "tri": False},
        # the benchmark's batch: uneven block sizes and horizons, solved again and again, autotuned once
        {"name": "batch 4096 mixed f32 tuned", "kind": "batch", "count": 4096, "ns": "6,12,14,24", "N0": 16, "N1": 128,
         "f64": False, "tuned": True, "sizes": 1},
        # a batch that is planned and run as it comes, odd block sizes among it
        {"name": "batch 600 odd f32", "kind": "batch", "count": 600, "ns": "4,7,13,14,21", "N0": 10, "N1": 100,
         "f64": False, "tuned": False, "sizes": 2},
        # FP64 systems of one robot, uneven horizons
        {"name": "batch 300 n14 f64", "kind": "batch", "count": 300, "ns": "14", "N0": 20, "N1": 64,
         "f64": True, "tuned": False, "sizes": 3},
        # from host memory and back: what a CPU-side program that forms S pays
        {"name": "batch host 1024 mixed f32", "kind": "batch_host", "count": 1024, "ns": "6,12,14,24", "N0": 16,
         "N1": 128, "f64": False, "sizes": 4},
        # a training step through the solver
        {"name": "pair 1024 n14 N64", "kind": "pair", "count": 1024, "n": 14, "N": 64},
        # the precision workload: ill-conditioned, to a true FP64 residual of 1e-10
        {"name": "refine 256 n24 N256", "kind": "refine", "count": 256, "n": 24, "N": 256},
        # the steps around a solve, for many short horizons or a long one at once
        {"name": "schur n24 m12 N65536 f32", "kind": "schur", "n": 24, "m": 12, "N": 65536, "f64": False, "pinv": True},
        {"name": "backsub n14 m7 N40001 f32", "kind": "backsub", "n": 14, "m": 7, "N": 40001, "f64": False},
        {"name": "jacobi 2048 mixed f32", "kind": "jacobi", "count": 2048, "ns": "6,12,14,24", "N0": 16, "N1": 128,
         "f64": False, "sizes": 5},
    ]


def _log_int(rng, lo, hi):
    return min(hi, max(lo, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    kind = rng.choice(["solve", "solve", "solve_host", "batch", "batch", "batch_host", "pair", "refine", "schur",
                       "schur", "backsub", "jacobi"])
    if kind in ("solve", "solve_host"):
        f64 = rng.random() < 0.4
        c = {"kind": kind, "n": rng.randint(2, 24), "N": _log_int(rng, 8, 256), "f64": f64, "tri": rng.random() < 0.5}
        if kind == "solve" and rng.random() < 0.3:  # a long horizon
            c.update(n=rng.randint(4, 16), N=_log_int(rng, 512, 8192), f64=False, tri=False)
        return c
    if kind in ("batch", "batch_host", "jacobi"):
        ns = sorted(rng.sample(range(2, 25), rng.choice([1, 2, 4])))
        N0 = rng.randint(8, 48)
        c = {"kind": kind, "count": _log_int(rng, 64, 1024), "ns": ",".join(map(str, ns)), "N0": N0,
             "N1": N0 + rng.randint(8, 64), "f64": kind != "batch_host" and rng.random() < 0.3,
             "sizes": rng.randint(10, 10 ** 6)}
        if kind == "batch":
            c["tuned"] = False
        return c
    if kind == "pair":
        return {"kind": kind, "count": _log_int(rng, 64, 1024), "n": rng.randint(3, 14), "N": rng.randint(16, 64)}
    if kind == "refine":
        return {"kind": kind, "count": _log_int(rng, 16, 256), "n": rng.randint(8, 24), "N": _log_int(rng, 32, 256)}
    f64 = rng.random() < 0.3
    n = rng.randint(2, 24)
    c = {"kind": kind, "n": n, "m": rng.randint(1, max(1, n // 2 + 2)), "N": _log_int(rng, 128, 30000 if f64 else 60000),
         "f64": f64}
    if kind == "schur":
        c["pinv"] = rng.random() < 0.6
    return c


# ------------------------------------------------------------------ problems
def _dtype(case):
    return torch.float64 if case.get("f64") or case["kind"] == "refine" else torch.float32


def _gen(seed):
    g = torch.Generator(device=DEV)
    g.manual_seed(int(seed) * 7919 + 17)
    return g


def _knots(n, m, K, g, ill=False):
    """A (K, n, n), B (K, n, m), Q (K, n), R (K, m) of K knots in 64 bits."""
    A = torch.randn(K, n, n, generator=g, device=DEV, dtype=torch.float64) / math.sqrt(n)
    B = torch.randn(K, n, m, generator=g, device=DEV, dtype=torch.float64)
    P = A
    for _ in range(6):
        P = P @ P
    A = A * (0.98 / P.square().sum((1, 2)).pow(1.0 / 128).clamp_min(1e-3))[:, None, None]
    u = torch.rand(K, n, generator=g, device=DEV, dtype=torch.float64)
    v = torch.rand(K, m, generator=g, device=DEV, dtype=torch.float64)
    if ill:
        return A, B, torch.exp(math.log(1e-2) + u * math.log(1e6)), torch.exp(math.log(1e-3) * (1 - v))
    return A, B, 1 + 9 * u, 0.1 + 0.9 * v


def _blocks(n, lengths, g, ill=False):
    """Diagonal blocks D (K, n, n) and sub-diagonal blocks L (K, n, n; zero at each
    system's first knot) of S for systems of `lengths` knots laid end to end."""
    m = max(1, n // 2)
    K = sum(lengths)
    ends = torch.tensor(np.cumsum(lengths), device=DEV)
    first = torch.zeros(K, dtype=torch.bool, device=DEV)
    first[0] = True
    first[ends[:-1]] = True
    A, B, Q, R = _knots(n, m, K + 1, g, ill)
    Qi, Ri = 1 / Q, 1 / R
    D = (A[:K] * Qi[:K, None, :]) @ A[:K].transpose(1, 2) + (B[:K] * Ri[:K, None, :]) @ B[:K].transpose(1, 2)
    D = D + torch.diag_embed(Qi[1:])
    D = 0.5 * (D + D.transpose(1, 2))
    L = -(A[:K] * Qi[:K, None, :])  # S_{k,k-1} = -A_k Q_k^-1
    L[first] = 0
    return D, L


def _rows(D, L, lengths):
    """Block rows (K, 3n, n): element (r, c) of block row k at [k, c, r]."""
    K, n, _ = D.shape
    S = torch.zeros(K, 3 * n, n, device=DEV, dtype=D.dtype)
    S[:, :n] = L.transpose(1, 2)
    S[:, n:2 * n] = D  # symmetric
    S[:-1, 2 * n:] = L[1:]  # (r, c) of S_{k,k+1} = L_{k+1}[c, r]
    return S


def _problem(case, seed):
    """A batch of systems in packed arenas: descs (n, N, offsets of S, Phi^-1 and the
    vectors, in elements, 16-byte aligned), S, gamma, sizes of the arenas."""
    dt = _dtype(case)
    g = _gen(seed)
    if "ns" in case:
        r = random.Random(case["sizes"])
        ns = [int(x) for x in case["ns"].split(",")]
        sizes = [(r.choice(ns), r.randint(case["N0"], case["N1"])) for _ in range(case["count"])]
    else:
        sizes = [(case["n"], case["N"])] * case.get("count", 1)
    al = 2 if dt == torch.float64 else 4
    up = lambda x: -(-x // al) * al  # noqa: E731
    descs, oS, oP, oV = [], 0, 0, 0
    for n, N in sizes:
        descs.append((n, N, oS, oP, oV))
        oS, oP, oV = oS + up(3 * n * n * N), oP + up(n * n * N), oV + up(n * N)
    S = torch.zeros(oS, device=DEV, dtype=dt)
    gamma = torch.zeros(oV, device=DEV, dtype=dt)
    for n in sorted(set(n for n, _ in sizes)):
        mine = [d for d in descs if d[0] == n]
        lengths = [d[1] for d in mine]
        rows = _rows(*_blocks(n, lengths, g, case["kind"] == "refine"), lengths).to(dt).reshape(-1)
        v = torch.randn(n * sum(lengths), generator=g, device=DEV, dtype=torch.float64).to(dt)
        at = 0
        for _, N, s, _, w in mine:
            S[s:s + 3 * n * n * N] = rows[3 * n * n * at:3 * n * n * (at + N)]
            gamma[w:w + n * N] = v[n * at:n * (at + N)]
            at += N
    return descs, S, gamma, oP


def _target(case, seed):
    g = _gen(seed + 1000003)
    return torch.randn(case["count"], case["n"] * case["N"], generator=g, device=DEV, dtype=torch.float32)


def _stages(case, seed):
    """Trajectory-optimisation data of N knots: A, B, Q, R, q, r, c and multipliers."""
    n, m, N, dt, g = case["n"], case["m"], case["N"], _dtype(case), _gen(seed)
    A, B, Q, R = _knots(n, m, N + 1, g)
    flat = lambda t: t.transpose(1, 2).contiguous().reshape(-1).to(dt)  # noqa: E731  (column-major blocks)
    vec = lambda k: torch.randn(k, generator=g, device=DEV, dtype=torch.float64).to(dt)  # noqa: E731
    return {"A": flat(A[:N]), "B": flat(B[:N]), "Qd": Q.reshape(-1).to(dt), "Rd": R[:N].reshape(-1).to(dt),
            "q": vec(n * (N + 1)), "r": vec(m * N), "c": vec(n * N), "lam": vec(n * N)}


# ------------------------------------------------------------------ states
_handles = {}


def _handle(key=None):
    """A program's handle; a tuned batch has one of its own, with its tuning table."""
    if key not in _handles:
        _handles[key] = gbdpcg.Handle(0)
    return _handles[key]


def _config(case):
    kind = case["kind"]
    if kind == "refine":
        return gbdpcg.config(exit_mode=gbdpcg.EXIT_RELRES, exit_tol=1e-10, max_iter=40000, max_outer=60, zero_guess=1)
    if kind in ("solve", "solve_host") and case["N"] <= 256:  # the reference's exit test
        return gbdpcg.config(max_iter=500, exit_tol=1e-12 if case["f64"] else 1e-6, zero_guess=1)
    return gbdpcg.config(max_iter=1000, exit_tol=1e-10 if case.get("f64") else 1e-6, exit_mode=gbdpcg.EXIT_RELRES,
                         zero_guess=1)


def prepare(case, seed):
    kind, dt = case["kind"], _dtype(case)
    s = {"case": case}
    if kind in ("schur", "backsub"):
        n, m, N = case["n"], case["m"], case["N"]
        s["in"] = _stages(case, seed)
        if kind == "schur":
            s["out"] = [torch.empty(3 * n * n * N, device=DEV, dtype=dt), torch.empty(n * N, device=DEV, dtype=dt)]
            s["pinv"] = torch.empty(n * n * N, device=DEV, dtype=dt) if case["pinv"] else None
        else:
            s["out"] = [torch.empty(n * (N + 1), device=DEV, dtype=dt), torch.empty(m * N, device=DEV, dtype=dt)]
        return s
    descs, S, gamma, oP = _problem(case, seed)
    s["cfg"] = cfg = _config(case)
    n, N = descs[0][:2]
    if kind in ("solve", "solve_host"):
        h = _handle()
        layout = gbdpcg.PINV_CBTD if case["tri"] else gbdpcg.PINV_BLOCKDIAG
        P = torch.empty((3 if case["tri"] else 1) * n * n * N, device=DEV, dtype=dt)
        h.block_jacobi(S, P, n, N, layout)
        if kind == "solve":
            s.update(h=h, S=S[:3 * n * n * N], P=P, gamma=gamma[:n * N], lam=torch.zeros_like(gamma[:n * N]), layout=layout)
        else:
            s.update(S=S[:3 * n * n * N].cpu().numpy(), P=P.cpu().numpy() if case["tri"] else None,
                     gamma=gamma[:n * N].cpu().numpy(), lam=np.zeros(n * N, np.float64 if case["f64"] else np.float32))
        return s
    if kind == "pair":
        P = torch.empty(oP, device=DEV, dtype=dt)
        lam, mu, dS, star = torch.zeros_like(gamma), torch.zeros_like(gamma), torch.zeros_like(S), _target(case, seed)
        sysl = [{"S": S[a:], "Pinv": P[b:], "gamma": gamma[v:], "lambda": lam[v:], "lambda_target": star[i],
                 "grad_gamma": mu[v:], "grad_S": dS[a:], "n": n, "N": N} for i, (n, N, a, b, v) in enumerate(descs)]
        h = _handle()
        for x in sysl:
            h.block_jacobi(x["S"], x["Pinv"], n, N)
        s.update(plan=gbdpcg.Plan.forward_adjoint(h, sysl, gbdpcg.PINV_BLOCKDIAG, cfg), keep=(S, P, gamma, star), out=[lam, mu, dS])
        return s
    lam = torch.zeros_like(gamma)
    if kind == "refine":
        P = torch.empty(oP, device=DEV, dtype=torch.float32)
        h = _handle()
        sysl = [{"S": S[a:], "Pinv": P[b:], "gamma": gamma[v:], "lambda": lam[v:], "n": n, "N": N}
                for n, N, a, b, v in descs]
        for x in sysl:
            h.block_jacobi_f64to32(x["S"], x["Pinv"], n, N)
        s.update(plan=gbdpcg.Plan(h, sysl, gbdpcg.PINV_BLOCKDIAG, cfg, dtype=2), keep=(S, P, gamma), lam=lam)
        return s
    P = torch.zeros(oP, device=DEV, dtype=dt)
    tuned = case.get("tuned", False)
    h = _handle(repr(sorted(case.items())) if tuned else None)
    plan = gbdpcg.Plan(h, layout=gbdpcg.PINV_BLOCKDIAG, cfg=cfg, packed=(descs, S, P, gamma, lam))
    if kind != "jacobi":
        plan.build_block_jacobi()
    if tuned and not h.tune_export():  # once; later plans of the handle take its table
        plan.autotune(gbdpcg.TUNE_RECURRENCE | gbdpcg.TUNE_WHOLE_PLAN)
    s.update(plan=plan, keep=(S, P, gamma), lam=lam, P=P)
    if kind == "batch_host":
        s["host"] = [t.cpu().pin_memory() for t in (S, gamma, lam)]
    return s


def run(s):
    case = s["case"]
    kind = case["kind"]
    if kind == "solve":
        s["h"].solve(s["S"], s["P"], s["gamma"], s["lam"], case["n"], case["N"], s["layout"], s["cfg"])
        return s["lam"]
    if kind == "solve_host":
        gbdpcg.solve(s["S"], s["P"], s["gamma"], s["lam"], case["n"], case["N"], s["cfg"])
        return s["lam"]
    if kind in ("batch", "refine"):
        s["plan"].execute()
        return s["lam"]
    if kind == "batch_host":
        s["plan"].solve_host(*s["host"], with_results=True)
        return s["host"][2]
    if kind == "pair":
        s["plan"].execute()
        return s["out"]
    if kind == "jacobi":
        s["plan"].build_block_jacobi()
        return s["P"]
    d, n, m, N = s["in"], case["n"], case["m"], case["N"]
    if kind == "schur":
        gbdpcg.form_schur(d["A"], d["B"], d["Qd"], d["Rd"], d["q"], d["r"], d["c"], n, m, N, *s["out"], Pinv_out=s["pinv"])
        return s["out"] + ([s["pinv"]] if s["pinv"] is not None else [])
    gbdpcg.kkt_backsub(d["A"], d["B"], d["Qd"], d["Rd"], d["q"], d["r"], d["lam"], n, m, N, *s["out"])
    return s["out"]


# ------------------------------------------------------------------ floors
def work(case):
    """Matrices and right-hand sides read once, results written once; the operations
    of the passes that such systems typically take to their tolerance."""
    kind, e = case["kind"], 8 if case.get("f64") or case["kind"] == "refine" else 4
    if kind in ("schur", "backsub"):
        n, m, N = case["n"], case["m"], case["N"]
        data = (n * n + n * m + 2 * n + 2 * m) * N + 2 * n
        if kind == "backsub":
            return {"bytes": e * (data + n * N + (n + m) * N + n), "flops": 2 * (n * n + n * m + 2 * n + 2 * m) * N}
        flops = (2 * (n + m) * n * n + 2 * n * n + 4 * (n + m) * n) * N
        out = 3 * n * n + n
        if case["pinv"]:
            flops, out = flops + 2 * n ** 3 * N, out + n * n
        return {"bytes": e * (data + n * N + out * N), "flops": flops}
    if "ns" in case:
        r = random.Random(case["sizes"])
        ns = [int(x) for x in case["ns"].split(",")]
        sizes = [(r.choice(ns), r.randint(case["N0"], case["N1"])) for _ in range(case["count"])]
    else:
        sizes = [(case["n"], case["N"])] * case.get("count", 1)
    passes = {"refine": 1000, "pair": 55}.get(kind, 40 if case.get("f64") else 25)
    total = {"bytes": 0, "flops": 0}
    for n, N in sizes:
        if kind == "jacobi":
            total["bytes"] += 2 * e * n * n * N
            total["flops"] += 2 * n ** 3 * N
            continue
        band = (3 * N - 2) * n * n
        pe = 4 if kind == "refine" else e
        total["bytes"] += e * (band + 2 * n * N) + pe * n * n * N * (3 if case.get("tri") else 1)
        total["flops"] += passes * (2 * band + 2 * n * n * N + 10 * n * N)
        if kind == "pair":
            total["bytes"] += e * (2 * n * N + 3 * n * n * N)
            total["flops"] += 4 * band
    return total


# ------------------------------------------------------------------ in 64 bits
def _factor(descs, S):
    """Block Cholesky of every system, systems of one block size together: the
    factors, and solve(vectors in the arena's layout) for them."""
    groups = []
    for n in sorted(set(d[0] for d in descs)):
        mine = sorted((d for d in descs if d[0] == n), key=lambda d: -d[1])
        Nmax = mine[0][1]
        D = torch.zeros(Nmax, len(mine), n, n, dtype=torch.float64, device=DEV)
        L = torch.zeros_like(D)
        for j, (_, N, s, _, _) in enumerate(mine):
            rows = S[s:s + 3 * n * n * N].reshape(N, 3 * n, n).double()
            D[:N, j] = rows[:, n:2 * n].transpose(1, 2)
            L[:N, j] = rows[:, :n].transpose(1, 2)
        live = [sum(1 for d in mine if d[1] > k) for k in range(Nmax)]
        for k in range(Nmax):
            a = live[k]
            if k:  # L_k C_{k-1}^-T, C the factors of the diagonal
                L[k, :a] = torch.linalg.solve_triangular(D[k - 1, :a], L[k, :a].transpose(1, 2), upper=False).transpose(1, 2)
                D[k, :a] -= L[k, :a] @ L[k, :a].transpose(1, 2)
            D[k, :a] = torch.linalg.cholesky_ex(D[k, :a])[0]
        groups.append((n, mine, live, D, L))

    def solve(v):
        out = torch.zeros_like(v, dtype=torch.float64)
        for n, mine, live, D, L in groups:
            X = torch.zeros(len(live), len(mine), n, 1, dtype=torch.float64, device=DEV)
            for j, (_, N, _, _, w) in enumerate(mine):
                X[:N, j, :, 0] = v[w:w + n * N].reshape(N, n).double()
            for k, a in enumerate(live):
                if k:
                    X[k, :a] -= L[k, :a] @ X[k - 1, :a]
                X[k, :a] = torch.linalg.solve_triangular(D[k, :a], X[k, :a], upper=False)
            for k in reversed(range(len(live))):
                a = live[k + 1] if k + 1 < len(live) else 0
                if a:
                    X[k, :a] -= L[k + 1, :a].transpose(1, 2) @ X[k + 1, :a]
                b = live[k]
                X[k, :b] = torch.linalg.solve_triangular(D[k, :b].transpose(1, 2), X[k, :b], upper=True)
            for j, (_, N, _, _, w) in enumerate(mine):
                out[w:w + n * N] = X[:N, j].reshape(-1)
        return out

    return solve


def exact(case, seed):
    kind = case["kind"]
    if kind in ("schur", "backsub"):
        n, m, N = case["n"], case["m"], case["N"]
        d = {k: v.double() for k, v in _stages(case, seed).items()}
        A, B = d["A"].reshape(N, n, n).transpose(1, 2), d["B"].reshape(N, m, n).transpose(1, 2)
        Q, R, q, r = d["Qd"].reshape(N + 1, n), d["Rd"].reshape(N, m), d["q"].reshape(N + 1, n), d["r"].reshape(N, m)
        if kind == "backsub":
            lam = d["lam"].reshape(N, n)
            x = q.clone()
            x[:N] += (A.transpose(1, 2) @ lam[:, :, None])[:, :, 0]
            x[1:] -= lam
            return [(-x / Q).reshape(-1), (-(r + (B.transpose(1, 2) @ lam[:, :, None])[:, :, 0]) / R).reshape(-1)]
        Qi, Ri = 1 / Q, 1 / R
        D = (A * Qi[:N, None, :]) @ A.transpose(1, 2) + (B * Ri[:, None, :]) @ B.transpose(1, 2) + torch.diag_embed(Qi[1:])
        L = -(A * Qi[:N, None, :])
        L[0] = 0
        gam = -(d["c"].reshape(N, n) + (A @ (Qi[:N] * q[:N])[:, :, None])[:, :, 0]
                + (B @ (Ri * r)[:, :, None])[:, :, 0] - Qi[1:] * q[1:])
        out = [_rows(D, L, [N]).reshape(-1), gam.reshape(-1)]
        return out + ([torch.linalg.inv(D).reshape(-1)] if case["pinv"] else [])
    descs, S, gamma, oP = _problem(case, seed)
    if kind == "jacobi":
        P = torch.zeros(oP, dtype=torch.float64, device=DEV)
        for n in sorted(set(d[0] for d in descs)):
            mine = [d for d in descs if d[0] == n]
            D = torch.cat([S[s:s + 3 * n * n * N].reshape(N, 3 * n, n)[:, n:2 * n] for _, N, s, _, _ in mine]).double()
            inv, at = torch.linalg.inv(D), 0
            for _, N, _, p, _ in mine:
                P[p:p + n * n * N] = inv[at:at + N].reshape(-1)
                at += N
        return P
    solve = _factor(descs, S)
    lam = solve(gamma)
    if kind != "pair":
        return lam[:case["n"] * case["N"]] if kind in ("solve", "solve_host") else lam
    n, N, cnt = case["n"], case["N"], case["count"]
    star = torch.zeros_like(lam)
    for (_, _, _, _, v), t in zip(descs, _target(case, seed)):
        star[v:v + n * N] = t.double()
    mu = solve(lam - star)
    dS = torch.zeros(S.numel(), dtype=torch.float64, device=DEV)
    for _, _, s, _, v in descs:
        l, u = lam[v:v + n * N].reshape(N, n), mu[v:v + n * N].reshape(N, n)
        rows = torch.zeros(N, 3 * n, n, dtype=torch.float64, device=DEV)
        outer = lambda a, b, x, y: -0.5 * (y[:, :, None] * a[:, None, :] + x[:, :, None] * b[:, None, :])  # noqa: E731
        rows[:, n:2 * n] = outer(u, l, u, l)
        rows[1:, :n] = outer(u[1:], l[1:], u[:-1], l[:-1])
        rows[:-1, 2 * n:] = outer(u[:-1], l[:-1], u[1:], l[1:])
        dS[s:s + 3 * n * n * N] = rows.reshape(-1)
    return [lam, mu, dS]
