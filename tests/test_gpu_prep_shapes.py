"""The fused Rytov preparation over resize ratios, odd maps, crops and non-finite pixels
against the per-pixel path (prepare_stack) followed by the transform in float64, and the
Ewald mapping's accumulation against a float64 scatter (wrapping and narrow plane ranges,
angle counts around the eight-angle step).  Tolerances: spectra 2e-6 relative L2 (one float32
transform); mapped data 2e-6 relative L2, hit counts equal."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m,n,r", [(16, 64, 64), (64, 64, 32), (65, 64, 64), (33, 70, 64), (100, 64, 64),
                                   (256, 1024, 512), (384, 384, 384), (2, 128, 128)])
@pytest.mark.parametrize("odd", [False, True])
def test_spectra_of_any_resize(ctx, dev, m, n, r, odd):
    import torch
    g = torch.Generator(device=dev).manual_seed(m * 1000 + n)
    a = 3
    ph = torch.randn((a, m, m), generator=g, device=dev) * 2
    am = torch.rand((a, m, m), generator=g, device=dev) + 0.5
    am[0, m // 2, m // 3] = 0.0
    am[1] *= -1
    if odd:
        ph[0, 0, 0], ph[1, m - 1, m // 2], am[0, m // 2, m - 1] = float("nan"), float("inf"), float("-inf")
        am[1, 0, m - 1], am[2, m // 2, m // 2] = float("nan"), 3.0e38
    U = torch.empty((a, r, r), dtype=torch.complex64, device=dev)
    p2, a2 = (torch.empty((a, r, r), device=dev) for _ in range(2))
    ctx.prepare_spectra(ph, am, U, a, m, n, r)
    ctx.prepare_stack(ph, am, p2, a2, a, m, n, r)
    u = torch.complex(torch.log(a2.double()), p2.double()).transpose(1, 2)
    ref = torch.fft.fft2(torch.roll(u, (r // 2, r // 2), (1, 2)))
    assert ((U - ref).norm() / ref.norm()).item() < 2e-6


@pytest.mark.parametrize("r,dx,angles,na", [(32, 4e-7, 1, 0.9), (64, 1e-7, 7, 0.9), (64, 4e-7, 8, 1.2),
                                            (128, 1e-7, 9, 0.0), (128, 2e-7, 33, 0.9), (384, 1e-7, 16, 0.9)])
def test_mapping_counts_and_values(ctx, dev, r, dx, angles, na):
    import torch
    n_med, lam = 1.337, 532e-9
    fm0, df = n_med / lam, 1.0 / (r * dx)
    phi = 2 * np.pi * np.arange(angles) / angles
    ax, ay = (np.arcsin(na / n_med * f(phi)).astype(np.float32) for f in (np.sin, np.cos))
    g = torch.Generator(device=dev).manual_seed(r + angles)
    U = torch.randn((angles, r, r), dtype=torch.complex64, generator=g, device=dev)
    F2 = torch.full((r, r, r), float("nan"), dtype=torch.complex64, device=dev)
    cnt = torch.full((r, r, r), -1, dtype=torch.int32, device=dev)
    ctx.map_ewald(U, ax, ay, fm0, df, dx, F2, cnt)
    s = np.fft.fftfreq(r, 1.0 / r)
    F, Cn = np.zeros((r, r, r), np.complex128), np.zeros((r, r, r), np.int64)
    iy, ix = np.mgrid[0:r, 0:r]
    for a in range(angles):
        fx0, fy0 = fm0 * np.sin(np.float64(ay[a])), fm0 * np.sin(np.float64(ax[a]))
        rad = fm0 * fm0 - (((s * df + fx0) ** 2)[None, :] + ((s * df + fy0) ** 2)[:, None])
        ok = rad >= 0
        fz = np.sqrt(np.where(ok, rad, 0))
        t = (fz - np.sqrt(fm0 * fm0 - fx0 * fx0 - fy0 * fy0)) / df
        nz = np.where(t > 0, np.floor(t + 0.5), np.ceil(t - 0.5)).astype(int) % r
        np.add.at(F, (nz[ok], iy[ok], ix[ok]), (4j * np.pi * fz * U[a].cpu().numpy())[ok])
        np.add.at(Cn, (nz[ok], iy[ok], ix[ok]), 1)
    ref = np.where(Cn > 0, F / np.maximum(Cn, 1), 0) / np.float64(np.float32(dx))
    assert np.array_equal(cnt.cpu().numpy(), Cn)
    assert np.linalg.norm(F2.cpu().numpy() - ref) / np.linalg.norm(ref) < 2e-6
