"""The gradient form's update at lambda = 0, handed over by the adjoint's last transform, at the
sides whose threads hold 16 and 24 points of a row (two and three eights): against FISTA in
float64 (torch).  Tolerance: contrasts after three updates 1e-5 RMS."""
import pytest

pytestmark = pytest.mark.gpu
K2 = 4.0


@pytest.mark.parametrize("positive", [False, True])
@pytest.mark.parametrize("r", [256, 384])
def test_update(dev, r, positive):
    import torch
    import ctdm_gb300 as C
    g = torch.Generator(device=dev).manual_seed(r)
    keep = torch.rand((r, r, r), generator=g, device=dev) < 0.1
    n = torch.randn((4, r, r, r), generator=g, device=dev)
    F2 = torch.where(keep, torch.complex(n[0], n[1]), 0).to(torch.complex64) * (-K2 * r ** 1.5 * 0.1)
    V = (0.1 * torch.complex(n[2], n[3])).contiguous()
    tape = C.Tape(F2.contiguous(), r, K2, keep.to(torch.int32).contiguous())
    data = F2.to(torch.complex128) / (-K2 * r ** 1.5)
    W = x = V.to(torch.complex128)
    t = 1.0
    for _ in range(3):
        res = torch.where(keep, torch.fft.fftn(W) / r ** 1.5 - data, 0)
        xn = W - torch.fft.ifftn(res) * r ** 1.5
        if positive:
            s = torch.sqrt(1 + xn)
            xn = torch.complex(s.real.clamp(min=1.0), s.imag.clamp(min=0.0)) ** 2 - 1
        tn = 0.5 * (1 + (1 + 4 * t * t) ** 0.5)
        W, x, t = xn + (t - 1) / tn * (xn - x), xn, tn
    v = V.clone()
    tape.reconstruct(v, 3, 0.0, positivity=positive)
    torch.cuda.synchronize()
    tape.close()
    assert (v - x).abs().square().mean().sqrt().item() <= 1e-5
