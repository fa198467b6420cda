"""alpha of FP32 systems with FP64 dot products is the correctly rounded quotient of
doubles rounded to float: systems of one equation S lambda = gamma whose quotient
gamma^2 / (gamma fl(S gamma)) lies within 2^-44 of the middle of two floats, beside
random ones.  One pass gives lambda = fl(alpha gamma), restated here bit for bit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

HARD = [("0x1.eba5180000000p+0", "0x1.afbf9a0000000p+1"), ("0x1.046c880000000p+0", "0x1.0c55d80000000p-1"),
        ("0x1.a2b4fc0000000p+0", "0x1.0ca7940000000p+1"), ("0x1.0c17620000000p+0", "0x1.2c20420000000p+0"),
        ("0x1.c661d80000000p+0", "0x1.959c3e0000000p+1")]


def test_alpha(gb, handle):
    import torch
    r = np.random.default_rng(3)
    f = np.float32
    g = np.concatenate([[float.fromhex(a) for a, _ in HARD], 1 + r.random(500), 2.0 ** r.integers(-30, 30, 500)]).astype(f)
    S = np.concatenate([[float.fromhex(b) for _, b in HARD], 0.5 + 3 * r.random(500), 1 + r.random(500)]).astype(f)
    wide = np.float64
    y = (S.astype(wide) * g).astype(f)
    alpha = (g.astype(wide) ** 2 / (g.astype(wide) * y)).astype(f)
    want = (alpha.astype(wide) * g).astype(f)
    rows = torch.zeros(len(g), 4, device="cuda")
    rows[:, 1] = torch.from_numpy(S).cuda()
    P, lam = torch.ones(len(g), 4, device="cuda"), torch.zeros(len(g), 4, device="cuda")
    gam = torch.zeros(len(g), 4, device="cuda")
    gam[:, 0] = torch.from_numpy(g).cuda()
    cfg = gb.config(max_iter=1, exit_tol=0.0, exit_mode=gb.EXIT_RELRES, zero_guess=1, dot_precision=gb.DOT_FP64)
    plan = gb.Plan(handle, [{"S": rows[i], "Pinv": P[i], "gamma": gam[i], "lambda": lam[i], "n": 1, "N": 1}
                            for i in range(len(g))], gb.PINV_BLOCKDIAG, cfg)
    plan.execute()
    torch.cuda.synchronize()
    plan.close()
    assert np.array_equal(lam[:, 0].cpu().numpy(), want)
