"""The DCT unwrap's error against 64 bits (scipy's DCT), on large maps of a noisy specimen and on
small maps of noise.  Bounds: what the 2M-point transforms of the mirrored lines gave on such
maps, mean relative L2 over 192 of the large ones 4.5, 5.6 and 9.0e-7 at 384, 512 and 768, over
320 of the small ones 2.2, 4.0 and 8.6e-6 at 64, 128 and 256, with 8% for another sample."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def wrapped(m, maps, rng):
    yy, xx = np.linspace(-1, 1, m)[:, None], np.linspace(-1, 1, m)[None, :]
    out = np.empty((maps, m, m), np.float32)
    for a in range(maps):
        u = rng.uniform(-1, 1, 5)
        p = 12 * np.maximum(1 - ((xx - 0.2 * u[0]) / 0.6) ** 2 - ((yy - 0.2 * u[1]) / 0.5) ** 2, 0)
        p = p + 2.4 * np.exp(-((xx - 0.3 * u[2]) ** 2 + (yy - 0.3 * u[3]) ** 2) / 0.02) + 0.5 * u[4] * xx
        p = p + 0.05 * rng.standard_normal((m, m))
        out[a] = p - 2 * np.pi * np.round(p / (2 * np.pi))
    return out


def unwrap64(phi):
    import scipy.fft as sf
    m = phi.shape[-1]
    p = phi.astype(np.float64)

    def wrap(t):
        return t - 2 * np.pi * np.round(t / (2 * np.pi))

    gx, gy = np.zeros_like(p), np.zeros_like(p)
    gx[..., :-1], gy[..., :-1, :] = wrap(np.diff(p, axis=-1)), wrap(np.diff(p, axis=-2))
    lap = gx + gy
    lap[..., 1:] -= gx[..., :-1]
    lap[..., 1:, :] -= gy[..., :-1, :]
    e = 4 * np.sin(2 * np.pi * np.arange(m) / (4 * m - 1)) ** 2
    d = -(e[:, None] + e[None, :])
    d[0, 0] = 1
    x = sf.dctn(lap, type=2, axes=(-2, -1), norm="ortho", workers=8) / d
    x[..., 0, 0] = 0
    return sf.idctn(x, type=2, axes=(-2, -1), norm="ortho", workers=8)


@pytest.mark.parametrize("m,mirrored", [(384, 4.5e-7), (512, 5.6e-7), (768, 9.0e-7)])
def test_error_of_large_maps(ctx, dev, m, mirrored):
    import torch
    err = []
    for seed in range(6):
        phi = wrapped(m, 16, np.random.default_rng([m, seed]))
        d = torch.from_numpy(phi).to(dev)
        out = torch.empty_like(d)
        ctx.unwrap_dct(d, out, 16, m, 1)
        ref = unwrap64(phi)
        err.append(np.linalg.norm(out.cpu().numpy() - ref) / np.linalg.norm(ref))
    assert np.mean(err) <= 1.08 * mirrored, err


@pytest.mark.parametrize("m,mirrored", [(64, 2.2e-6), (128, 4.0e-6), (256, 8.6e-6)])
def test_error_of_noise(ctx, dev, m, mirrored):
    import torch
    err = []
    for seed in range(40):
        phi = (1.5 * np.random.default_rng([m, seed]).standard_normal((8, m, m))).astype(np.float32)
        d = torch.from_numpy(phi).to(dev)
        out = torch.empty_like(d)
        ctx.unwrap_dct(d, out, 8, m, 1)
        ref = unwrap64(phi)
        err.append(np.linalg.norm(out.cpu().numpy() - ref) / np.linalg.norm(ref))
    assert np.mean(err) <= 1.08 * mirrored, err
