"""Odd block sizes with two rows a thread (an empty last row a knot): every on-chip
storage, both iteration forms, clusters of 1 to 8 CTAs with boundary knots on both
sides, batches with odd and even sizes in one launch, forward + adjoint pairs, and
guards around lambda (nothing is written past it).

The storages sum in the same order, so lambda is the same bit for bit at one cluster
and CTA size; accuracy against the 64-bit solution within 1.5 times (recurrence form:
3 times) the oracle's own error plus 1e-6, passes within one."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def relerr(a, b):
    return float(np.linalg.norm(np.asarray(a, np.float64) - b) / np.linalg.norm(b))


@pytest.mark.parametrize("n,N,C", [(1, 9, 1), (3, 50, 1), (5, 31, 2), (7, 64, 3), (9, 40, 1), (11, 55, 4), (13, 36, 1),
                                   (13, 120, 8), (15, 33, 2), (17, 20, 1), (21, 48, 5), (23, 20, 1), (23, 65, 7)])
def test_storages(gb, oracle_mod, handle, n, N, C):
    import torch
    O = oracle_mod
    sy = O.generate(n, N, 31 * n + N)
    S, P, g = sy.cbtd(np.float32), O.block_jacobi(sy.D, "compact").astype(np.float32), sy.gamma.astype(np.float32)
    x = O.block_cholesky_solve(S.astype(np.float64), n, N, g.astype(np.float64))
    lam_o, it_o = O.pcg(S, P, g, np.zeros(n * N, np.float32), n, N, 300, 1e-6, flags=O.PINV_BLOCKDIAG | O.EXIT_RELRES)[:2]
    tS, tP, tg = (torch.from_numpy(a).cuda() for a in (S, P, g))
    got = {}
    for alg in (gb.ALGO_AUTO, gb.ALGO_RECURRENCE):
        for storage in (gb.STORAGE_SPLIT, gb.STORAGE_TMEM, gb.STORAGE_HYBRID):
            guard = torch.full((n * N + 64,), 7.0, device="cuda")
            lam = guard[32:32 + n * N]
            cfg = gb.config(max_iter=300, exit_tol=1e-6, exit_mode=gb.EXIT_RELRES, zero_guess=1, algorithm=alg,
                            storage=storage, cluster_size=C)
            plan = gb.Plan(handle, [{"S": tS, "Pinv": tP, "gamma": tg, "lambda": lam, "n": n, "N": N}], gb.PINV_BLOCKDIAG, cfg)
            l = plan.launches()[0]
            plan.execute()
            r = plan.results()[0]
            plan.close()
            assert r.status == gb.CONVERGED and abs(int(r.iters) - it_o) <= 1 and l["rows_per_thread"] == 2, (r, l)
            assert bool((guard[:32] == 7).all()) and bool((guard[32 + n * N:] == 7).all())
            assert relerr(lam.cpu().numpy(), x) <= (1.5 if alg == gb.ALGO_AUTO else 3) * relerr(lam_o, x) + 1e-6
            key = (alg, l["cluster"], l["threads"])
            assert torch.equal(got.setdefault(key, lam.clone()), lam)


def test_mixed_launch(gb, oracle_mod, handle):
    """n = 13 and 14 share a kernel and its launches."""
    import torch
    O = oracle_mod
    cfg = gb.config(max_iter=300, exit_mode=gb.EXIT_RELRES, zero_guess=1)
    systems, alone = [], []
    for i in range(200):
        n, N = (13, 60) if i % 2 else (14, 60)
        sy = O.generate(n, N, i % 6)
        t = [torch.from_numpy(a.astype(np.float32)).cuda() for a in (sy.cbtd(np.float32), O.block_jacobi(sy.D, "compact"), sy.gamma)]
        systems.append({"S": t[0], "Pinv": t[1], "gamma": t[2], "lambda": torch.zeros_like(t[2]), "n": n, "N": N})
    plan = gb.Plan(handle, systems, gb.PINV_BLOCKDIAG, cfg)
    assert len(plan.launches()) == 1
    plan.execute()
    assert all(r.status == gb.CONVERGED for r in plan.results())
    plan.close()
    for s in systems[:12]:
        one = dict(s, **{"lambda": torch.zeros_like(s["lambda"])})
        p1 = gb.Plan(handle, [one], gb.PINV_BLOCKDIAG, cfg)
        p1.execute()
        torch.cuda.synchronize()
        assert torch.equal(one["lambda"], s["lambda"])
        p1.close()


@pytest.mark.parametrize("n,N", [(5, 20), (13, 40), (13, 90)])
def test_pair_and_adjoint(gb, oracle_mod, handle, n, N):
    """The pair against a dense FP64 gradient: relative errors within 1e-4 at an exit
    tolerance of 1e-7 (as for even n)."""
    import torch
    O = oracle_mod
    sy = O.generate(n, N, 3)
    S = torch.from_numpy(sy.cbtd(np.float32)).cuda()
    P = torch.from_numpy(O.block_jacobi(sy.D, "compact").astype(np.float32)).cuda()
    g = torch.from_numpy(sy.gamma.astype(np.float32)).cuda()
    star = torch.randn(n * N, generator=torch.Generator().manual_seed(5)).cuda()
    lam, mu, dS = torch.zeros_like(g), torch.zeros_like(g), torch.full_like(S, float("nan"))
    cfg = gb.config(max_iter=500, exit_tol=1e-7, exit_mode=gb.EXIT_RELRES, zero_guess=1)
    plan = gb.Plan.forward_adjoint(handle, [{"S": S, "Pinv": P, "gamma": g, "lambda": lam, "lambda_target": star,
                                             "grad_gamma": mu, "grad_S": dS, "n": n, "N": N}], gb.PINV_BLOCKDIAG, cfg)
    plan.execute()
    torch.cuda.synchronize()
    plan.close()
    S64 = S.cpu().numpy().astype(np.float64)
    x = O.block_cholesky_solve(S64, n, N, g.cpu().numpy().astype(np.float64))
    m = O.block_cholesky_solve(S64, n, N, x - star.cpu().numpy())
    assert relerr(lam.cpu().numpy(), x) < 1e-4 and relerr(mu.cpu().numpy(), m) < 1e-4
    X, Mu = x.reshape(N, n), m.reshape(N, n)
    want = np.zeros((N, 3, n, n))  # [k, block, column, row]
    for b in range(3):
        for k in range(N):
            j = k + b - 1
            if 0 <= j < N:
                want[k, b] = -0.5 * (np.outer(X[j], Mu[k]) + np.outer(Mu[j], X[k]))
    assert relerr(dS.cpu().numpy(), want.reshape(-1)) < 1e-4
