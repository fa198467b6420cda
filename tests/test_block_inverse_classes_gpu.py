"""Batches whose block-size classes go to both kernels of the builder: large classes
(8192 knots or more, four rows a lane) with small ones before, between and behind them
in the order of sizes, in one launch a run of small classes.  Every system's Phi^-1 is,
bit for bit, the one it gets alone, and nothing is written outside it."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("layout", ["compact", "cbtd"])
@pytest.mark.parametrize("large", [(8,), (16,), (32,), (8, 32), (12, 24), (8, 16, 32), (12, 16, 24), (6, 10, 14, 20)])
def test_runs(gb, handle, large, layout):
    import torch
    lay, w = (gb.PINV_CBTD, 3) if layout == "cbtd" else (gb.PINV_BLOCKDIAG, 1)
    g = torch.Generator(device="cuda").manual_seed(sum(large))
    sizes = [(n, N) for n in (5, 8, 11, 12, 13, 16, 20, 24, 29, 32) for N in (1, 37)] + [(n, 8192 // 40 + 3) for n in large for _ in range(40)]
    perm = torch.randperm(len(sizes), generator=torch.Generator().manual_seed(7)).tolist()
    systems, want = [], []
    for n, N in (sizes[i] for i in perm):
        a = torch.randn(N, n, n, device="cuda", generator=g)
        S = torch.zeros(N, 3, n, n, device="cuda")
        S[:, 1] = a @ a.transpose(1, 2) + n * torch.eye(n, device="cuda")
        S[:, 1] = 0.5 * (S[:, 1] + S[:, 1].transpose(1, 2))
        alone = torch.empty(w * n * n * N, device="cuda")
        handle.block_jacobi(S, alone, n, N, lay)
        guard = torch.full((w * n * n * N + 64,), 7.0, device="cuda")
        v = torch.zeros(n * N, device="cuda")
        systems.append({"S": S, "Pinv": guard[32:], "gamma": v, "lambda": v, "n": n, "N": N, "guard": guard})
        want.append(alone)
    plan = gb.Plan(handle, systems, lay, gb.config(zero_guess=1))
    plan.build_block_jacobi()
    torch.cuda.synchronize()
    plan.close()
    for s, p in zip(systems, want):
        assert torch.equal(s["guard"][32:32 + p.numel()], p)
        assert bool((s["guard"][:32] == 7).all()) and bool((s["guard"][32 + p.numel():] == 7).all())
