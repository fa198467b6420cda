"""Reductions of doubles (one warp per value sums the CTA's rows, pcg_cluster.cuh
onewarp_send / onewarp_finish) at the edges of their shapes: CTAs of 1 warp to
the most a kernel takes, odd numbers of warps, clusters of 1 to 16 CTAs, both
iteration forms, FP64 systems and FP32 systems with FP64 dots.

Bounds as for the FP64 solver elsewhere: the oracle's pass count and lambda
within 1e-12 at an exit tolerance of 1e-12; the recurrence form within one pass
and 3 times the oracle's error against the 64-bit solution; FP32 systems within one pass and
1.5 times the oracle's own error (plus 1e-6) against the 64-bit solution."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def relerr(a, b):
    return float(np.linalg.norm(np.asarray(a, np.float64) - b) / np.linalg.norm(b))


def _solve(gb, O, handle, n, N, f64, cfg, seed):
    import torch
    dt = np.float64 if f64 else np.float32
    sy = O.generate(n, N, seed)
    S, P, g = sy.cbtd(dt), O.block_jacobi(sy.D, "compact").astype(dt), sy.gamma.astype(dt)
    d = [torch.from_numpy(x).cuda() for x in (S, P, g, np.zeros(n * N, dt))]
    sysl = [{"S": d[0], "Pinv": d[1], "gamma": d[2], "lambda": d[3], "n": n, "N": N}]
    plan = gb.Plan(handle, sysl, gb.PINV_BLOCKDIAG, cfg)
    launch = plan.launches()[0]
    plan.execute()
    r = plan.results()[0]
    lam = d[3].cpu().numpy()
    plan.close()
    return S, P, g, launch, r.iters, lam


# n, N, cluster size, warps per CTA
SHAPES = [(4, 8, 1, 1), (4, 8, 4, 1), (6, 5, 1, 2), (3, 30, 1, 3), (8, 36, 1, 9), (8, 56, 2, 7), (6, 50, 3, 4),
          (7, 64, 5, 3), (14, 64, 8, 4), (14, 112, 16, 4), (2, 250, 1, 16)]


@pytest.mark.parametrize("alg", ["standard", "recurrence"])
@pytest.mark.parametrize("n,N,C,W", SHAPES)
def test_fp64_shapes(gb, oracle_mod, n, N, C, W, alg):
    O = oracle_mod
    h = gb.Handle(0)
    a = gb.ALGO_RECURRENCE if alg == "recurrence" else gb.ALGO_AUTO
    # rows in shared memory, one per thread: any number of warps
    h.tune_import(f"1 0 1 0 0 {a} 0 {n} {N} : 2 1 {3 if a else 0} {C} {32 * W}\n")
    cfg = gb.config(max_iter=300, exit_tol=1e-12, zero_guess=1, algorithm=a)
    S, P, g, launch, iters, lam = _solve(gb, O, h, n, N, True, cfg, n + N)
    assert (launch["cluster"], launch["threads"]) == (C, 32 * W), launch
    lam_o, it_o = O.pcg(S, P, g, np.zeros(n * N), n, N, 300, 1e-12, flags=O.PINV_BLOCKDIAG)[:2]
    if alg == "standard":
        assert iters == it_o
        assert relerr(lam, lam_o) < 1e-12
    else:  # iterates differ at roundoff level
        x = O.block_cholesky_solve(S, n, N, g)
        assert abs(int(iters) - it_o) <= 1
        assert relerr(lam, x) <= 3 * relerr(lam_o, x) + 1e-12
    h.close()


@pytest.mark.parametrize("n,N,C", [(6, 40, 1), (9, 40, 2), (14, 90, 5)])
def test_fp32_with_fp64_dots(gb, oracle_mod, handle, n, N, C):
    O = oracle_mod
    cfg = gb.config(max_iter=300, exit_tol=1e-6, zero_guess=1, cluster_size=C, dot_precision=gb.DOT_FP64)
    S, P, g, launch, iters, lam = _solve(gb, O, handle, n, N, False, cfg, n + N)
    assert launch["cluster"] == C
    lam_o, it_o = O.pcg(S, P, g, np.zeros(n * N, np.float32), n, N, 300, 1e-6,
                        flags=O.PINV_BLOCKDIAG | O.ACC64)[:2]
    x = O.block_cholesky_solve(S.astype(np.float64), n, N, g.astype(np.float64))
    assert abs(int(iters) - it_o) <= 1
    assert relerr(lam, x) <= 1.5 * relerr(lam_o, x) + 1e-6
