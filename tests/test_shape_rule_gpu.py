"""The storage rule of batches on both sides of its lines: tensor memory where the
other storage's CTA fills its SM or where the whole batch runs at once, split
rows where several of their CTAs share an SM, neither for odd n, FP64 or a cbtd
Phi^-1.  Both storages sum in the same order, so at the same cluster and CTA size
lambda is the same bit for bit; each is checked against the 64-bit solution at
the accuracy of the split rows."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SPLIT, TMEM = 1, 4


def _solve(gb, O, handle, n, N, count, storage):
    import torch
    sy = O.generate(n, N, 7 * n + N)
    S = torch.from_numpy(sy.cbtd(np.float32)).cuda()
    P = torch.from_numpy(O.block_jacobi(sy.D, "compact").astype(np.float32)).cuda()
    g = torch.from_numpy(sy.gamma.astype(np.float32)).cuda()
    lams = torch.full((count, n * N), float("nan"), device="cuda")
    cfg = gb.config(max_iter=300, exit_tol=1e-6, exit_mode=gb.EXIT_RELRES, zero_guess=1, storage=storage)
    plan = gb.Plan(handle, [{"S": S, "Pinv": P, "gamma": g, "lambda": lams[i], "n": n, "N": N} for i in range(count)],
                   gb.PINV_BLOCKDIAG, cfg)
    plan.execute()
    assert all(r.status == gb.CONVERGED for r in plan.results())
    l = plan.launches()[0]
    plan.close()
    assert bool((lams == lams[0]).all())
    x = O.block_cholesky_solve(S.cpu().numpy().astype(np.float64), n, N, g.cpu().numpy().astype(np.float64))
    lam = lams[0].cpu().numpy()
    return l, lam, float(np.linalg.norm(lam - x) / np.linalg.norm(x))


@pytest.mark.parametrize("n,N,count,want", [
    (14, 36, 400, TMEM), (14, 27, 400, SPLIT), (14, 27, 152, TMEM), (14, 27, 153, SPLIT), (14, 60, 100, TMEM),
    (24, 64, 76, TMEM), (24, 64, 300, TMEM), (24, 10, 300, SPLIT), (8, 64, 300, SPLIT), (8, 96, 300, TMEM),
    (6, 128, 300, TMEM), (6, 85, 300, SPLIT), (2, 3, 1, TMEM), (13, 36, 400, TMEM), (13, 27, 400, SPLIT),
    (23, 64, 300, TMEM), (7, 96, 300, TMEM), (7, 40, 400, SPLIT), (1, 5, 1, TMEM)])
def test_rule(gb, oracle_mod, handle, n, N, count, want):
    l, lam, err = _solve(gb, oracle_mod, handle, n, N, count, gb.STORAGE_AUTO)
    assert l["storage"] == want, l
    ls, lam_s, err_s = _solve(gb, oracle_mod, handle, n, N, 1, gb.STORAGE_SPLIT)
    if (l["cluster"], l["threads"]) == (ls["cluster"], ls["threads"]):
        assert np.array_equal(lam, lam_s)
    assert err <= 1.5 * err_s + 1e-6


def test_no_tensor_memory_for_fp64_or_cbtd(gb, oracle_mod, handle):
    import torch
    O = oracle_mod
    for n, dt, layout in ((14, np.float64, "compact"), (14, np.float32, "cbtd"), (13, np.float64, "compact")):
        sy = O.generate(n, 36, 3)
        t = [torch.from_numpy(a.astype(dt)).cuda() for a in (sy.cbtd(dt), O.block_jacobi(sy.D, layout), sy.gamma)]
        lam = torch.zeros_like(t[2])
        plan = gb.Plan(handle, [{"S": t[0], "Pinv": t[1], "gamma": t[2], "lambda": lam, "n": n, "N": 36}],
                       gb.PINV_CBTD if layout == "cbtd" else gb.PINV_BLOCKDIAG, gb.config(zero_guess=1))
        assert plan.launches()[0]["storage"] != TMEM
        plan.close()
