"""The line passes with empty columns left out: every y plan (8 or 16 lines per CTA) at the
sides that have several, and plans pinned by another thread while calls are enqueued (a call
reads its plans once).  Reference: the loop in float64 (torch).  Tolerance: the path's RI
bound, RMSE <= 1e-5."""
import threading

import pytest

pytestmark = pytest.mark.gpu
NM, K2 = 1.337, 1.0e14


def case(torch, dev, r):
    g = torch.Generator(device=dev).manual_seed(r)
    s = torch.fft.fftfreq(r, 1.0 / r, device=dev)
    disc = torch.hypot(s[:, None], s[None, :]) < 0.3 * r
    keep = disc[None] & (torch.rand((r, r, r), generator=g, device=dev) < 0.1)
    f = torch.zeros((r, r, r), dtype=torch.float64, device=dev)
    f[r // 6:r // 2, r // 4:3 * r // 4, r // 5:2 * r // 3] = 0.05
    F2 = torch.where(keep, torch.fft.fftn(-K2 * f), 0)
    noise = torch.randn((2, r, r, r), generator=g, device=dev)
    F2 = torch.where(keep, F2 + 0.02 * F2.abs().square().mean().sqrt() * torch.complex(noise[0], noise[1]), 0)
    return keep, F2.to(torch.complex64)


def loop64(torch, F2, keep, iters):
    def est(v):
        n = NM * torch.sqrt(1 - v / K2)
        return torch.complex(n.real.clamp(min=NM), n.imag.clamp(min=0.0))

    d = F2.to(torch.complex128)
    v = torch.fft.ifftn(d)
    for _ in range(iters):
        v = torch.fft.ifftn(torch.where(keep, d, torch.fft.fftn(-K2 * ((est(v) / NM) ** 2 - 1))))
    return torch.roll(est(v), (F2.shape[0] // 2,) * 3, (0, 1, 2))


def rmse(out, ref):
    return (out - ref).abs().square().mean().sqrt().item()


@pytest.mark.parametrize("r", [256, 384, 512, 768])
def test_every_y_plan(ctx, dev, r):
    import torch
    import ctdm_gb300 as C
    keep, F2 = case(torch, dev, r)
    ref = loop64(torch, F2, keep, 2)
    plans, scheme = C.plans(r)[0], C.loop_scheme(r)
    out = torch.empty_like(F2)
    try:
        C.set_loop_scheme(r, 0)
        for v in range(3):
            C.set_plans(r, (0, v, (v + 1) % 3))
            ctx.positivity(F2, r, 2, K2, NM, out)
            torch.cuda.synchronize()
            assert rmse(out, ref) <= 1e-5, v
    finally:
        C.set_plans(r, plans)
        C.set_loop_scheme(r, scheme)


def test_plans_pinned_meanwhile(ctx, dev):
    import torch
    import ctdm_gb300 as C
    r = 256
    keep, F2 = case(torch, dev, r)
    ref = loop64(torch, F2, keep, 3)
    plans, scheme = C.plans(r)[0], C.loop_scheme(r)
    out = torch.empty_like(F2)
    done = threading.Event()

    def pin():
        i = 0
        while not done.is_set():
            C.set_plans(r, (i % 3, i // 2 % 3, i % 3))
            C.set_loop_scheme(r, 0 if i % 5 else 1)
            i += 1

    t = threading.Thread(target=pin)
    t.start()
    try:
        for _ in range(30):
            ctx.positivity(F2, r, 3, K2, NM, out)
            torch.cuda.synchronize()
            assert rmse(out, ref) <= 1e-5
    finally:
        done.set()
        t.join()
        C.set_plans(r, plans)
        C.set_loop_scheme(r, scheme)
