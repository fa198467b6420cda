"""Threads that launch one kernel with different amounts of shared memory: no call may
lower the limit under another's launch, which would then be refused."""
import threading

import pytest

pytestmark = pytest.mark.gpu


def _hammer(works, calls):
    """Runs each work `calls` times on a thread and stream of its own; the errors."""
    import torch
    errors, ready = [], threading.Barrier(len(works))

    def go(work):
        st = torch.cuda.Stream()
        ready.wait()
        for _ in range(calls):
            try:
                work(st.cuda_stream)
            except RuntimeError as e:
                errors.append(e)
    threads = [threading.Thread(target=go, args=(w,)) for w in works]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    torch.cuda.synchronize()
    return errors


def test_formation(gb):
    """n = 32 with m = 1 and with m = 32 and Phi^-1: on both sides of the default limit."""
    import torch

    def work(m):
        n, N = 32, 4
        g = torch.Generator(device="cuda").manual_seed(m)
        src = [torch.rand(k, device="cuda", generator=g) + 0.5 for k in
               (n * n * N, n * m * N, n * (N + 1), m * N, n * (N + 1), m * N, n * N)]
        out = [torch.empty(k, device="cuda", dtype=torch.float32) for k in (3 * n * n * N, n * N, n * n * N)]
        src, out = [t.double() for t in src], [t.double() for t in out]
        return lambda st: gb.form_schur(*src, n, m, N, *out[:2], Pinv_out=out[2], stream=st)
    works = [work(m) for m in (1, 32, 8, 24)]
    torch.cuda.synchronize()
    errors = _hammer(works, 2000)
    assert not errors, (len(errors), errors[0])


def test_long_systems(gb):
    """The whole-GPU kernel with 50 and 95 KB a CTA, on a handle a thread."""
    import torch

    def work(N):
        h = gb.Handle(0)
        S = torch.zeros(N, 3, device="cuda")
        S[:, 1] = 2
        P, g, lam = torch.zeros(N, 3, device="cuda"), torch.ones(N, device="cuda"), torch.zeros(N, device="cuda")
        P[:, 1] = 0.5
        cfg = gb.config(max_iter=1, exit_mode=gb.EXIT_RELRES, zero_guess=1)
        return lambda st: h.solve(S, P, g, lam, 1, N, gb.PINV_CBTD, cfg, stream=st, sync=False)
    works = [work(N) for N in (160000, 300000)]
    torch.cuda.synchronize()
    errors = _hammer(works, 1500)
    assert not errors, (len(errors), errors[0])
