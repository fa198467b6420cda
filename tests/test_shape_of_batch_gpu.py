"""A system's cluster and CTA size do not depend on the batch around it: alone in a
plan (where tensor memory may take the split rows' place, which gives the same bits)
and among 152 others, at every block size over the range of horizons; and the same
lambda, bit for bit, from a whole plan and from the pieces of a host pipeline."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", range(1, 33))
def test_shape(gb, handle, n):
    import torch
    buf = torch.zeros(3 * n * n * 200, device="cuda")
    cfg = gb.config(zero_guess=1)
    for N in sorted(set(int(round(2 ** (i / 4))) for i in range(31)) | {27, 72, 73}):
        one = {"S": buf, "Pinv": buf, "gamma": buf, "lambda": buf, "n": n, "N": N}
        shapes = []
        for count in (1, 153):
            plan = gb.Plan(handle, [one] * count, gb.PINV_BLOCKDIAG, cfg)  # (made, not run)
            shapes.append([(l["cluster"], l["threads"]) for l in plan.launches()])
            plan.close()
        assert shapes[0] == shapes[1], (n, N, shapes)


@pytest.mark.parametrize("n,N,count", [(14, 27, 200), (24, 72, 300), (13, 40, 240), (20, 100, 160), (8, 64, 300), (6, 128, 200)])
def test_pieces(gb, oracle_mod, handle, n, N, count):
    import torch
    O = oracle_mod
    sys_, S, P, g = [O.generate(n, N, i) for i in range(4)], [], [], []
    for i in range(count):
        sy = sys_[i % 4]
        S.append(sy.cbtd(np.float32))
        P.append(O.block_jacobi(sy.D, "compact").astype(np.float32))
        g.append(sy.gamma.astype(np.float32))
    up = lambda x: -(-x // 4) * 4  # noqa: E731
    sizes = [up(a[0].size) for a in (S, P, g)]
    arenas = []
    for a, w in zip((S, P, g), sizes):
        t = np.zeros(w * count, np.float32)
        for i, x in enumerate(a):
            t[i * w:i * w + x.size] = x.reshape(-1)
        arenas.append(t)
    descs = [(n, N, i * sizes[0], i * sizes[1], i * sizes[2]) for i in range(count)]
    out = []
    for pieces in (1, 4):
        dev = [torch.zeros(a.size, device="cuda") for a in arenas] + [torch.zeros(arenas[2].size, device="cuda")]
        cfg = gb.config(max_iter=300, exit_tol=1e-6, exit_mode=gb.EXIT_RELRES, zero_guess=1, host_pieces=pieces)
        plan = gb.Plan(handle, layout=gb.PINV_BLOCKDIAG, cfg=cfg, packed=(descs, *dev))
        lam = np.zeros(arenas[2].size, np.float32)
        assert all(r.status == gb.CONVERGED for r in plan.execute_host(*arenas, lam, with_results=True))
        out.append(lam)
        plan.close()
    assert out[0].tobytes() == out[1].tobytes()
