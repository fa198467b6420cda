"""The whole-GPU kernel of one long system (pcg_grid.cuh) at the edges of its
ranges: rows of S in registers, streamed with one and with two rows a thread,
blocks narrower than their bound, one knot a CTA, both layouts of Phi^-1, both
precisions; warm starts, exhausted budgets, captured streams (which take the
cluster kernel) and solves on two streams at once.

Bounds against the streamed-row cluster kernel on the same system, whose sums
run in another order: FP64 the same passes and lambda within 1e-12; FP32 within
one pass, and 1.5 times its error against the 64-bit solution plus 1e-6."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def relerr(a, b):
    return float(np.linalg.norm(np.asarray(a, np.float64) - b) / np.linalg.norm(b))


def _system(O, n, N, f64, layout):
    import torch
    dt = np.float64 if f64 else np.float32
    sy = O.generate(n, N, n + N)
    S, P, g = sy.cbtd(dt), O.block_jacobi(sy.D, layout).astype(dt), sy.gamma.astype(dt)
    return S, g, [torch.from_numpy(a).cuda() for a in (S, P, g)]


# n, N, FP64, layout: what the CTAs get with 152 SMs
CASES = [(14, 1500, False, "compact"), (14, 8192, False, "compact"),  # 10 and 54 knots, rows in registers
         (14, 9000, False, "compact"), (14, 12000, False, "compact"),  # streamed, one and two rows a thread
         (13, 1500, False, "compact"), (23, 800, False, "compact"), (32, 500, False, "compact"),
         (6, 5000, False, "compact"), (5, 6001, False, "compact"),
         (14, 700, False, "cbtd"), (9, 3001, False, "cbtd"), (24, 300, False, "cbtd"), (32, 330, False, "cbtd"),
         (14, 500, True, "compact"), (24, 200, True, "compact"), (7, 2000, True, "compact"), (32, 152, True, "compact"),
         (24, 100, True, "cbtd"), (14, 4000, True, "cbtd"), (32, 90, True, "cbtd")]


@pytest.mark.parametrize("n,N,f64,layout", CASES)
def test_against_streamed_rows(gb, oracle_mod, handle, n, N, f64, layout):
    import torch
    O = oracle_mod
    S, g, (tS, tP, tg) = _system(O, n, N, f64, layout)
    lay = gb.PINV_CBTD if layout == "cbtd" else gb.PINV_BLOCKDIAG
    got = []
    for storage in (gb.STORAGE_AUTO, gb.STORAGE_STREAM):
        lam = torch.full_like(tg, float("nan"))
        cfg = gb.config(max_iter=400, exit_tol=1e-10 if f64 else 1e-6, exit_mode=gb.EXIT_RELRES, zero_guess=1,
                        storage=storage)
        r = handle.solve(tS, tP, tg, lam, n, N, lay, cfg)
        assert r.status == gb.CONVERGED, (storage, r)
        got.append((r.iters, lam.cpu().numpy()))
    (it, lam), (it_s, lam_s) = got
    if f64:
        assert it == it_s and relerr(lam, lam_s) < 1e-12
    else:
        x = O.block_cholesky_solve(S.astype(np.float64), n, N, g.astype(np.float64))
        assert abs(int(it) - int(it_s)) <= 1
        assert relerr(lam, x) <= 1.5 * relerr(lam_s, x) + 1e-6


def test_is_the_route(gb, oracle_mod, handle):
    """It is what AUTO takes: a pinned cluster size gives other bits at n=14 N=1500."""
    import torch
    _, _, (tS, tP, tg) = _system(oracle_mod, 14, 1500, False, "compact")
    lams = []
    for c in (0, 16):
        lam = torch.zeros_like(tg)
        handle.solve(tS, tP, tg, lam, 14, 1500, gb.PINV_BLOCKDIAG,
                     gb.config(max_iter=400, exit_mode=gb.EXIT_RELRES, cluster_size=c))
        lams.append(lam)
    assert not torch.equal(*lams)


@pytest.mark.parametrize("f64,layout", [(False, "compact"), (True, "cbtd")])
def test_warm_start_budget_and_zero_rhs(gb, oracle_mod, handle, f64, layout):
    import torch
    n, N = 14, 800 if f64 else 1500
    _, _, (tS, tP, tg) = _system(oracle_mod, n, N, f64, layout)
    lay = gb.PINV_CBTD if layout == "cbtd" else gb.PINV_BLOCKDIAG
    kw = dict(exit_tol=1e-10 if f64 else 1e-6, exit_mode=gb.EXIT_RELRES)
    lam = torch.zeros_like(tg)
    full = handle.solve(tS, tP, tg, lam, n, N, lay, gb.config(max_iter=400, **kw))
    # in two legs from where the first stopped: converged, with at least the passes of one leg
    legs = torch.zeros_like(tg)
    r = handle.solve(tS, tP, tg, legs, n, N, lay, gb.config(max_iter=7, **kw))
    assert (r.status, r.iters) == (gb.MAX_ITER, 7)
    r = handle.solve(tS, tP, tg, legs, n, N, lay, gb.config(max_iter=400, **kw))
    assert r.status == gb.CONVERGED and 7 + r.iters >= full.iters
    # no pass allowed: lambda stays the guess
    keep = lam.clone()
    r = handle.solve(tS, tP, tg, lam, n, N, lay, gb.config(max_iter=0, **kw))
    assert r.iters == 0 and torch.equal(lam, keep)
    # zero right-hand side: alpha = 0 and one pass
    lam.zero_()
    r = handle.solve(tS, tP, torch.zeros_like(tg), lam, n, N, lay, gb.config(max_iter=400, **kw))
    assert r.iters == 1 and not lam.any()


def test_two_streams_and_capture(gb, oracle_mod, handle):
    import torch
    n, N = 14, 1500
    cfg = gb.config(max_iter=400, exit_mode=gb.EXIT_RELRES, zero_guess=1)
    sysl = [_system(oracle_mod, n, N + i, False, "compact")[2] for i in range(2)]
    alone = []
    for i, (tS, tP, tg) in enumerate(sysl):
        lam = torch.zeros_like(tg)
        handle.solve(tS, tP, tg, lam, n, N + i, gb.PINV_BLOCKDIAG, cfg)
        alone.append(lam)
    torch.cuda.synchronize()
    streams = [torch.cuda.Stream() for _ in sysl]
    for _ in range(5):
        lams = [torch.zeros_like(s[2]) for s in sysl]
        torch.cuda.synchronize()
        for i, (st, (tS, tP, tg)) in enumerate(zip(streams, sysl)):
            handle.solve(tS, tP, tg, lams[i], n, N + i, gb.PINV_BLOCKDIAG, cfg, stream=st, sync=False)
        torch.cuda.synchronize()
        assert all(torch.equal(a, b) for a, b in zip(lams, alone))
    # under capture: replays solve, to the accuracy of the others
    tS, tP, tg = sysl[0]
    lam = torch.zeros_like(tg)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        handle.solve(tS, tP, tg, lam, n, N, gb.PINV_BLOCKDIAG, cfg, sync=False)
    lam.zero_()
    graph.replay()
    torch.cuda.synchronize()
    assert relerr(lam.cpu().numpy(), alone[0].cpu().numpy().astype(np.float64)) < 1e-5


def test_host_arrays(gb, oracle_mod, handle):
    """A host call of such a system stages its arrays: lambda as from device arrays, bit for bit."""
    import torch
    n, N = 14, 700
    S, g, (tS, tP, tg) = _system(oracle_mod, n, N, False, "cbtd")
    cfg = gb.config(max_iter=400, exit_mode=gb.EXIT_RELRES)
    lam = np.zeros(n * N, np.float32)
    r = gb.solve(S, tP.cpu().numpy(), g, lam, n, N, cfg)
    dev = torch.zeros_like(tg)
    assert handle.solve(tS, tP, tg, dev, n, N, gb.PINV_CBTD, cfg).iters == r.iters
    assert np.array_equal(lam, dev.cpu().numpy())
