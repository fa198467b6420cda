"""Block inverses of blocks that are not positive definite: negative definite,
indefinite, singular and nearly singular ones, and definite ones whose diagonal
spans many powers of two.  Both kernels of the builder (four rows a lane from 8192
knots of a class on), the plan's builder and the fused formation give, bit for bit,
what elimination without pivoting gives when it divides the pivot row: restated here
on the CPU, with every fused multiply-add rounded once (FP32 through FP64, FP64
through the 113-bit long double of the host)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

LD = np.longdouble


def _eliminate(D):
    """Inverses of the blocks D (K, n, n): Gauss-Jordan without pivoting, a zero pivot
    taken as 1, averaged with the transpose."""
    dt = D.dtype.type
    wide = np.float64 if dt is np.float32 else LD
    a = D.copy()
    with np.errstate(all="ignore"):
        for j in range(D.shape[1]):
            piv = a[:, j, j].copy()
            piv[piv == 0] = 1
            inv = dt(1) / piv
            t = a[:, j, :] * inv[:, None]
            t[:, j] = inv
            m = a[:, :, j].copy()
            a = (a.astype(wide) - m.astype(wide)[:, :, None] * t.astype(wide)[:, None, :]).astype(dt)
            a[:, :, j] = -(m * inv[:, None])
            a[:, j, :] = t
        return dt(0.5) * (a + a.transpose(0, 2, 1))


def _blocks(kind, n, K, dt, seed):
    r = np.random.default_rng(seed)
    a = r.standard_normal((K, n, n))
    spd = a @ a.transpose(0, 2, 1) / n + 0.3 * np.eye(n)
    if kind == "negative":
        d = -spd
    elif kind == "indefinite":
        d = a + a.transpose(0, 2, 1)
    elif kind == "one negative":  # a positive first diagonal element, one negative eigenvalue
        d = spd.copy()
        d[:, n - 1, n - 1] -= 3 * np.abs(spd[:, n - 1, n - 1])
    elif kind == "singular":  # exact zero pivots
        v = r.integers(1, 3, (K, n, 1)).astype(np.float64)
        d = 4 * v @ v.transpose(0, 2, 1)
    elif kind == "nearly singular":
        v = r.standard_normal((K, n, 1))
        d = v @ v.transpose(0, 2, 1) + (1e-7 if dt is np.float32 else 1e-16) * np.eye(n)
    else:  # scales
        s = 2.0 ** r.integers(-15, 16, (K, n, 1))
        d = s * spd * s.transpose(0, 2, 1)
    d = d.astype(dt)
    return np.triu(d) + np.triu(d, 1).transpose(0, 2, 1)


KINDS = ["negative", "indefinite", "one negative", "singular", "nearly singular", "scales"]


def _rows(D, N):
    import torch
    n = D.shape[1]
    S = torch.zeros(N, 3, n, n, dtype=torch.from_numpy(D[:1]).dtype, device="cuda")
    S[:, 1] = torch.from_numpy(D).cuda()[torch.arange(N, device="cuda") % len(D)]
    return S.reshape(-1)


def _same(P, want, N):
    import torch
    w = torch.from_numpy(want).cuda()[torch.arange(N, device="cuda") % len(want)].reshape(-1)
    assert torch.equal(torch.isnan(P), torch.isnan(w))
    assert torch.equal(torch.nan_to_num(P), torch.nan_to_num(w))


@pytest.mark.parametrize("kind", KINDS)
@pytest.mark.parametrize("n", [1, 5, 8, 9, 12, 14, 16, 21, 24, 29, 32])
def test_fp32(gb, handle, n, kind):
    import torch
    D = _blocks(kind, n, 23, np.float32, 7 * n)
    want = _eliminate(D)
    for N in (1, 61, 8209):  # one row a lane; four rows a lane from 8192 on
        S = _rows(D, N)
        P = torch.full((n * n * N,), 7.0, device="cuda")
        handle.block_jacobi(S, P, n, N)
        _same(P, want, N)
        T = torch.full((3 * n * n * N,), 7.0, device="cuda")
        handle.block_jacobi(S, T, n, N, gb.PINV_CBTD)
        T = T.reshape(N, 3, n * n)
        _same(T[:, 1].reshape(-1), want, N)
        assert not T[:, 0].any() and not T[:, 2].any()


@pytest.mark.skipif(np.finfo(LD).nmant < 106, reason="no 113-bit long double on this host")
@pytest.mark.parametrize("kind", KINDS)
@pytest.mark.parametrize("n", [1, 7, 8, 12, 14, 24, 32])
def test_fp64(gb, handle, n, kind):
    import torch
    D = _blocks(kind, n, 5, np.float64, 7 * n)
    want = _eliminate(D)
    N = 13
    S = _rows(D, N)
    P = torch.full((n * n * N,), 7.0, device="cuda", dtype=torch.float64)
    handle.block_jacobi(S, P, n, N)
    _same(P, want, N)
    P32 = torch.full((n * n * N,), 7.0, device="cuda")
    handle.block_jacobi_f64to32(S, P32, n, N)
    with np.errstate(all="ignore"):
        _same(P32, want.astype(np.float32), N)


def test_plan_with_single_blocks_among_many(gb, handle):
    """One indefinite block a system, at a random knot: it and its neighbours in the warp are right."""
    import torch
    systems, wants = [], []
    r = np.random.default_rng(5)
    for i in range(400):
        n, N = [(6, 45), (14, 40), (24, 50), (32, 7), (12, 30)][i % 5]
        D = _blocks("scales", n, N, np.float32, i)
        D[r.integers(N)] = _blocks("indefinite", n, 1, np.float32, 1000 + i)[0]
        wants.append(_eliminate(D))
        g = torch.zeros(n * N, device="cuda")
        systems.append({"S": _rows(D, N), "Pinv": torch.full((n * n * N,), 7.0, device="cuda"), "gamma": g, "lambda": g.clone(),
                        "n": n, "N": N})
    assert sum(s["N"] for s in systems if s["n"] == 14) < 8192
    plan = gb.Plan(handle, systems * 3, gb.PINV_BLOCKDIAG, gb.config(zero_guess=1))  # n=24: 12000 knots, four rows a lane
    plan.build_block_jacobi()
    torch.cuda.synchronize()
    plan.close()
    for s, w in zip(systems, wants):
        _same(s["Pinv"], w, s["N"])


@pytest.mark.parametrize("f64", [False, True])
@pytest.mark.parametrize("n,m,N", [(3, 2, 9), (8, 4, 33), (14, 7, 4101), (24, 12, 19), (32, 8, 6)])
def test_formation(gb, handle, n, m, N, f64):
    """Phi^-1 of the formation for costs of either sign: of the negated costs the
    negative, and for mixed signs what the builder makes of the S it formed."""
    import torch
    dt = torch.float64 if f64 else torch.float32
    g = torch.Generator(device="cuda").manual_seed(n * 100 + m)
    rnd = lambda k: torch.randn(k, device="cuda", generator=g, dtype=dt)  # noqa: E731
    pos = lambda k: 0.5 + torch.rand(k, device="cuda", generator=g, dtype=dt)  # noqa: E731
    A, B, Q, R = rnd(n * n * N), rnd(n * m * N), pos(n * (N + 1)), pos(m * N)
    rest = [rnd(n * (N + 1)), rnd(m * N), rnd(n * N)]

    def form(Q, R):
        out = [torch.full((k,), 7.0, device="cuda", dtype=dt) for k in (3 * n * n * N, n * N, n * n * N)]
        gb.form_schur(A, B, Q, R, *rest, n, m, N, *out[:2], Pinv_out=out[2])
        return out
    S, _, P = form(Q, R)
    Sn, _, Pn = form(-Q, -R)
    assert torch.equal(Sn, -S) and torch.equal(Pn, -P)
    Sm, _, Pm = form(torch.where(rnd(Q.numel()) < 0, -Q, Q), R)
    built = torch.empty_like(Pm)
    handle.block_jacobi(Sm, built, n, N)
    assert torch.equal(Pm, built)
