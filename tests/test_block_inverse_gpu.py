"""The block inverses of the block-Jacobi builder and the fused Schur formation at
the edges of their groups: every block-size class with n below, at and above its
bounds, fewer knots than a warp inverts at once and ragged ends, batches with the
classes mixed, both kernels (four rows a lane from 8192 knots of a class on), both
layouts, and arrays that are only element-aligned.

Both kernels and the formation run one elimination, so their results agree bit for
bit; against 64 bits the bound is Gauss-Jordan's, 10 n u cond(S_kk) with u = 2^-24
(2^-53), doubled for the residual growth of the unpivoted elimination."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _blocks(O, n, N, seed):
    return O.generate(n, N, seed)


def _check(D, P, n, N, f64):
    u = 2.0 ** -53 if f64 else 2.0 ** -24
    D = D.astype(np.float64 if f64 else np.float32).astype(np.float64)
    P = P.reshape(N, n, n).astype(np.float64)
    assert np.array_equal(P, P.transpose(0, 2, 1))
    for d, p in zip(D, P):
        x = np.linalg.inv(d)
        assert np.linalg.norm(p - x) <= 20 * n * u * np.linalg.cond(d) * np.linalg.norm(x)


@pytest.mark.parametrize("f64", [False, True])
@pytest.mark.parametrize("n,N", [(1, 5), (2, 1), (7, 3), (8, 17), (9, 2), (12, 11), (13, 1), (16, 9), (17, 6), (24, 7), (25, 3),
                                 (32, 5)])
def test_single_system(gb, oracle_mod, handle, n, N, f64):
    import torch
    dt = np.float64 if f64 else np.float32
    sy = _blocks(oracle_mod, n, N, 10 * n + N)
    S = torch.from_numpy(sy.cbtd(dt)).cuda()
    P = torch.full((n * n * N,), float("nan"), device="cuda", dtype=S.dtype)
    handle.block_jacobi(S, P, n, N)
    _check(sy.D, P.cpu().numpy(), n, N, f64)
    T = torch.full((3 * n * n * N,), float("nan"), device="cuda", dtype=S.dtype)
    handle.block_jacobi(S, T, n, N, gb.PINV_CBTD)
    rows = T.reshape(N, 3, n * n)
    assert torch.equal(rows[:, 1].reshape(-1), P) and not rows[:, 0].any() and not rows[:, 2].any()


@pytest.mark.parametrize("layout", ["compact", "cbtd"])
@pytest.mark.parametrize("n", [5, 6, 8, 10, 12, 14, 15, 16, 21, 22, 24, 31, 32])
def test_many_knots_equal_few(gb, oracle_mod, handle, n, layout):
    """N = 8209 takes four rows a lane; the same blocks in a short system one. Element-aligned arrays too."""
    import torch
    N, M = 8209, 61
    sy = _blocks(oracle_mod, n, M, n)
    rows = torch.from_numpy(sy.cbtd(np.float32)).cuda().reshape(M, -1)
    S = rows[torch.arange(N, device="cuda") % M].reshape(-1)
    lay, w = (gb.PINV_CBTD, 3) if layout == "cbtd" else (gb.PINV_BLOCKDIAG, 1)
    few = torch.empty(w * n * n * M, device="cuda")
    handle.block_jacobi(rows.reshape(-1), few, n, M, lay)
    want = few.reshape(M, -1)[torch.arange(N, device="cuda") % M].reshape(-1)
    for shift in (0, 1, 2):  # 16-, 4- and 8-byte alignment
        pad = torch.empty(S.numel() + 4, device="cuda")
        s = pad[shift:shift + S.numel()].copy_(S)
        out = torch.full((w * n * n * N + 4,), float("nan"), device="cuda")[shift:shift + w * n * n * N]
        handle.block_jacobi(s, out, n, N, lay)
        assert torch.equal(out, want), shift


@pytest.mark.parametrize("scale", [1, 60])
def test_mixed_batch(gb, oracle_mod, handle, scale):
    """Classes side by side in one plan; with 60 copies some take four rows a lane."""
    import torch
    O = oracle_mod
    sizes = [(6, 20), (24, 33), (14, 64), (3, 7), (12, 41), (32, 2), (9, 30), (20, 16), (14, 90), (5, 55)]
    systems, want = [], []
    for i, (n, N) in enumerate(sizes):
        sy = _blocks(O, n, N, 500 + i)
        S = torch.from_numpy(sy.cbtd(np.float32)).cuda()
        one = torch.empty(n * n * N, device="cuda")
        handle.block_jacobi(S, one, n, N)
        for _ in range(scale):
            g = torch.zeros(n * N, device="cuda")
            systems.append({"S": S, "Pinv": torch.full_like(one, float("nan")), "gamma": g, "lambda": g.clone(), "n": n, "N": N})
            want.append(one)
    plan = gb.Plan(handle, systems, gb.PINV_BLOCKDIAG, gb.config(zero_guess=1))
    plan.build_block_jacobi()
    torch.cuda.synchronize()
    assert all(torch.equal(s["Pinv"], w) for s, w in zip(systems, want))
    plan.close()


@pytest.mark.parametrize("n,m,N", [(1, 1, 1), (7, 2, 5), (8, 8, 33), (13, 6, 3), (14, 7, 130), (16, 1, 9), (24, 12, 17), (32, 32, 6)])
def test_formation_alignments(gb, oracle_mod, n, m, N):
    """S, gamma and Phi^-1 are the same bits from arrays of every alignment (accesses of 16, 8 and 4 bytes)."""
    import torch
    g = torch.Generator(device="cuda").manual_seed(n * 100 + m)
    rnd = lambda k: torch.randn(k, device="cuda", generator=g)  # noqa: E731
    pos = lambda k: 0.5 + torch.rand(k, device="cuda", generator=g)  # noqa: E731
    src = [rnd(n * n * N), rnd(n * m * N), pos(n * (N + 1)), pos(m * N), rnd(n * (N + 1)), rnd(m * N), rnd(n * N)]
    got = []
    for shift in (0, 2, 1):
        ins = [torch.empty(t.numel() + 4, device="cuda")[shift:shift + t.numel()].copy_(t) for t in src]
        outs = [torch.full((k + 4,), float("nan"), device="cuda")[shift:shift + k] for k in (3 * n * n * N, n * N, n * n * N)]
        gb.form_schur(*ins, n, m, N, outs[0], outs[1], outs[2])
        alone = [torch.empty_like(outs[0]), torch.empty_like(outs[1])]
        gb.form_schur(*ins, n, m, N, *alone)
        assert torch.equal(alone[0], outs[0]) and torch.equal(alone[1], outs[1])
        got.append([o.clone() for o in outs])
    for o in got[1:]:
        assert all(torch.equal(a, b) for a, b in zip(got[0], o))


@pytest.mark.parametrize("f64", [False, True])
@pytest.mark.parametrize("n,m,N", [(1, 1, 1), (5, 3, 9), (6, 3, 130), (8, 8, 3), (12, 12, 21), (13, 6, 2), (14, 7, 65), (16, 9, 5),
                                   (22, 11, 7), (24, 1, 4), (32, 32, 3)])
def test_back_substitution_alignments(gb, oracle_mod, n, m, N, f64):
    """x and u are the same bits from arrays of every alignment, and within the rounding of
    a sum of n + 2 terms and a division, (n + 4) u relative to the terms, of the 64-bit result."""
    import torch
    dt = torch.float64 if f64 else torch.float32
    g = torch.Generator(device="cuda").manual_seed(n * 100 + m)
    rnd = lambda k: torch.randn(k, device="cuda", generator=g, dtype=dt)  # noqa: E731
    pos = lambda k: 0.5 + torch.rand(k, device="cuda", generator=g, dtype=dt)  # noqa: E731
    src = [rnd(n * n * N), rnd(n * m * N), pos(n * (N + 1)), pos(m * N), rnd(n * (N + 1)), rnd(m * N), rnd(n * N)]
    got = []
    for shift in (0, 2, 1):
        ins = [torch.empty(t.numel() + 4, device="cuda", dtype=dt)[shift:shift + t.numel()].copy_(t) for t in src]
        x, u = (torch.full((k,), float("nan"), device="cuda", dtype=dt) for k in (n * (N + 1), m * N))
        gb.kkt_backsub(*ins, n, m, N, x, u)
        got.append((x, u))
    assert all(torch.equal(a, b) for o in got[1:] for a, b in zip(got[0], o))
    A, B, Q, R, q, r, lam = (t.double() for t in src)
    A, B, L = A.reshape(N, n, n), B.reshape(N, m, n), lam.reshape(N, n)  # [knot, column, row]
    xs, ax = q.reshape(N + 1, n).clone(), q.reshape(N + 1, n).abs()
    xs[:N] += (A @ L[:, :, None])[:, :, 0]
    ax[:N] += (A.abs() @ L.abs()[:, :, None])[:, :, 0]
    xs[1:] -= L
    ax[1:] += L.abs()
    us = r.reshape(N, m) + (B @ L[:, :, None])[:, :, 0]
    au = r.reshape(N, m).abs() + (B.abs() @ L.abs()[:, :, None])[:, :, 0]
    eps = 2.0 ** -53 if f64 else 2.0 ** -24
    for v, w, a, d in ((got[0][0], xs, ax, Q), (got[0][1], us, au, R)):
        w, a = -w.reshape(-1) / d, a.reshape(-1) / d
        # (the 64-bit reference rounds as often as an FP64 result)
        assert bool(((v.double() - w).abs() <= (2 if f64 else 1) * (n + 4) * eps * a).all())
