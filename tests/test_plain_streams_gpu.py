"""Plain solves of one handle on several streams take turns in the handle's scratch:
each gives the bits of the same solve alone, whatever is in flight around it, and so
do solves after a captured one."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_streams_take_turns(gb, oracle_mod, handle):
    import torch
    O = oracle_mod
    cfg = gb.config(max_iter=100, exit_mode=gb.EXIT_RELRES, zero_guess=1, algorithm=gb.ALGO_PLAIN)
    systems = []
    for i, (n, N) in enumerate([(5, 40), (14, 60), (6, 150), (14, 30)]):
        sy = O.generate(n, N, i)
        t = [torch.from_numpy(a.astype(np.float32)).cuda() for a in (sy.cbtd(np.float32), O.block_jacobi(sy.D, "cbtd"), sy.gamma)]
        lam = torch.zeros_like(t[2])
        assert handle.solve(*t, lam, n, N, gb.PINV_CBTD, cfg).status == gb.CONVERGED
        systems.append((n, N, t, lam))
    torch.cuda.synchronize()
    streams = [torch.cuda.Stream() for _ in systems]

    def overlap():
        lams = [torch.full_like(s[3], float("nan")) for s in systems]
        torch.cuda.synchronize()
        for _ in range(5):
            for st, (n, N, t, _), lam in zip(streams, systems, lams):
                handle.solve(*t, lam, n, N, gb.PINV_CBTD, cfg, stream=st, sync=False)
        torch.cuda.synchronize()
        assert all(torch.equal(lam, s[3]) for lam, s in zip(lams, systems))

    overlap()
    n, N, t, want = systems[1]
    lam, graph = torch.zeros_like(want), torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        handle.solve(*t, lam, n, N, gb.PINV_CBTD, cfg, sync=False)
    graph.replay()
    torch.cuda.synchronize()
    assert torch.equal(lam, want)
    overlap()
