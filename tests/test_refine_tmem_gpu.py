"""Refinement with its rows in tensor memory (pcg_refine.cuh, ST_TMEM): every
block-size bound, one and several CTAs a system, both kinds of inner dot
products; the shape rule of a batch; and the exact widening of the factors of
FP64 dots, by a power-of-two scaling of the right-hand side.

Bound: the exit test is on the true FP64 residual, so 1.2e-10 for a tolerance of
1e-10 (the residual of the returned lambda is summed in another order)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _plan(gb, O, handle, n, N, count, cfg, scale=1.0):
    import torch
    systems, host = [], []
    for i in range(count):
        sy = O.generate(n, N, 100 * n + i, ill=True)
        S = torch.from_numpy(sy.cbtd()).cuda()
        systems.append({"S": S, "Pinv": torch.empty(n * n * N, dtype=torch.float32, device="cuda"),
                        "gamma": torch.from_numpy(sy.gamma * scale).cuda(),
                        "lambda": torch.zeros(n * N, dtype=torch.float64, device="cuda"), "n": n, "N": N})
        host.append(sy)
    plan = gb.Plan(handle, systems, gb.PINV_BLOCKDIAG, cfg, dtype=2)
    plan.build_block_jacobi()
    plan.execute()
    return plan, systems, host


def _cfg(gb, **kw):
    return gb.config(exit_mode=gb.EXIT_RELRES, exit_tol=1e-10, max_iter=40000, max_outer=60, zero_guess=1, **kw)


@pytest.mark.parametrize("dot", ["fp64", "float2"])
@pytest.mark.parametrize("n,N,C", [(2, 9, 1), (6, 40, 2), (8, 33, 1), (10, 30, 3), (14, 54, 1), (16, 17, 2), (20, 40, 2),
                                   (24, 32, 1), (24, 65, 5)])
def test_tmem_refinement(gb, oracle_mod, handle, n, N, C, dot):
    O = oracle_mod
    cfg = _cfg(gb, storage=gb.STORAGE_TMEM, cluster_size=C,
               dot_precision=gb.DOT_FLOAT2 if dot == "float2" else gb.DOT_FP64)
    plan, systems, host = _plan(gb, O, handle, n, N, 3, cfg)
    l = plan.launches()[0]
    assert (l["storage"], l["cluster"]) == (4, C)
    for s, r, sy in zip(systems, plan.results(), host):
        assert r.status == gb.CONVERGED
        assert O.relres(sy.cbtd(), s["lambda"].cpu().numpy(), sy.gamma, n, N) <= 1.2e-10
    plan.close()


@pytest.mark.parametrize("n,N,storage", [(24, 64, 4), (14, 32, 4), (8, 32, 1), (13, 32, 0)])
def test_shape_rule(gb, oracle_mod, handle, n, N, storage):
    """Tensor memory where the other storage's CTA fills its SM; not where several fit, nor for odd n."""
    plan, systems, host = _plan(gb, oracle_mod, handle, n, N, 2, _cfg(gb))
    assert plan.launches()[0]["storage"] == storage
    plan.close()


@pytest.mark.parametrize("storage", ["STORAGE_TMEM", "STORAGE_SPLIT"])
def test_scaled_rhs_scales_lambda(gb, oracle_mod, handle, storage):
    """Every operation of the solve commutes with a scaling by 2^-60 that keeps its
    values normal: the same passes, and lambda scaled bit for bit."""
    out = []
    for scale in (1.0, 2.0 ** -60):
        plan, systems, _ = _plan(gb, oracle_mod, handle, 12, 24, 1, _cfg(gb, storage=getattr(gb, storage)), scale)
        r = plan.results()[0]
        out.append((r.iters, r.outer, systems[0]["lambda"].cpu().numpy() / scale))
        plan.close()
    assert out[0][:2] == out[1][:2]
    assert np.array_equal(out[0][2], out[1][2])
