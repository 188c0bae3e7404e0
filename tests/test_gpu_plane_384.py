"""The 384^3 loop on its plane passes (8- and 6-CTA clusters, radix-6 stages) and line passes
against the same loop in float64 (torch).  Tolerance: the path's RI bound, RMSE <= 1e-5."""
import pytest

pytestmark = pytest.mark.gpu
NM, K2, R = 1.337, 1.0e14, 384


@pytest.mark.parametrize("accelerated", [False, True])
@pytest.mark.parametrize("scheme", [0, 1, 2])
def test_loop_384(ctx, dev, scheme, accelerated):
    import torch
    import ctdm_gb300 as C
    g = torch.Generator(device=dev).manual_seed(scheme)
    s = torch.fft.fftfreq(R, 1.0 / R, device=dev)
    keep = (torch.hypot(s[:, None], s[None, :]) < 0.3 * R)[None] & (torch.rand((R, R, R), generator=g, device=dev) < 0.1)
    f = torch.zeros((R, R, R), dtype=torch.float64, device=dev)
    f[60:200, 100:300, 80:250] = 0.05
    F2 = torch.where(keep, torch.fft.fftn(-K2 * f), 0)
    noise = torch.randn((2, R, R, R), generator=g, device=dev)
    F2 = torch.where(keep, F2 + 0.02 * F2.abs().square().mean().sqrt() * torch.complex(noise[0], noise[1]), 0)
    F2 = F2.to(torch.complex64)

    def est(v):
        n = NM * torch.sqrt(1 - v / K2)
        return torch.complex(n.real.clamp(min=NM), n.imag.clamp(min=0.0))

    d = F2.to(torch.complex128)
    v, prev, t = torch.fft.ifftn(d), None, 1.0
    for _ in range(2):
        x = -K2 * ((est(v) / NM) ** 2 - 1)
        tn = 0.5 * (1 + (1 + 4 * t * t) ** 0.5)
        w = x + (t - 1) / tn * (x - prev) if accelerated and prev is not None else x
        prev, t = x, tn
        v = torch.fft.ifftn(torch.where(keep, d, torch.fft.fftn(w)))
    ref = torch.roll(est(v), (R // 2,) * 3, (0, 1, 2))
    saved = C.loop_scheme(R)
    out = torch.empty((R, R, R), dtype=torch.complex64, device=dev)
    try:
        C.set_loop_scheme(R, scheme)
        ctx.positivity(F2, R, 2, K2, NM, out, accelerated=accelerated)
        torch.cuda.synchronize()
    finally:
        C.set_loop_scheme(R, saved)
    assert (out - ref).abs().square().mean().sqrt().item() <= 1e-5
