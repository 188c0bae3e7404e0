"""The positivity loop on measured data that cover few z tiles: tiles (and, on the line
passes, x columns) without a measured voxel are left out of the transforms.  Reference:
the same loop over the whole volume in float64 numpy.  Tolerance: the path's RI bound,
RMSE <= 1e-5."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
NM, K2 = 1.337, 1.0e14


def loop64(F2, keep, iters, accelerated):
    def est(f):
        n = NM * np.sqrt(1.0 - f / K2)
        return np.maximum(n.real, NM) + 1j * np.maximum(n.imag, 0.0)

    f = np.fft.ifftn(F2)
    prev, t = None, 1.0
    for _ in range(iters):
        x = ((est(f) / NM) ** 2 - 1.0) * -K2
        tn = 0.5 * (1 + np.sqrt(1 + 4 * t * t))
        w = x + (t - 1) / tn * (x - prev) if accelerated and prev is not None else x
        prev, t = x, tn
        F = np.fft.fftn(w)
        F[keep] = F2[keep]
        f = np.fft.ifftn(F)
    return np.roll(est(f), (F2.shape[0] // 2,) * 3, (0, 1, 2))


def voxels(r, cover, rng):
    """Hit mask [z][y][x]: none, one voxel in the last tile, single tiles at the ends of a
    row, a disc of lateral frequencies (the caps' shape), every column."""
    m = np.zeros((r, r, r), bool)
    if cover == "corner":
        m[r - 1, r - 1, r - 1] = True
    elif cover == "ends":
        m[1, 3, 0] = m[2, 3, r - 1] = m[0, 0, 7] = m[5, r - 2, 8] = True
    elif cover == "disc":
        s = np.fft.fftfreq(r, 1.0 / r)
        d = np.hypot(s[:, None], s[None, :]) < 0.3 * r
        m[rng.integers(0, r, 3)[:, None], np.nonzero(d)[0], np.nonzero(d)[1]] = True
    elif cover == "all":
        m[rng.random((r, r, r)) < 0.05] = True
        m[0] = True
    return m


@pytest.mark.parametrize("cover", ["none", "corner", "ends", "disc", "all"])
@pytest.mark.parametrize("r,scheme", [(64, 0), (128, 0), (256, 0), (256, 1), (256, 2)])
def test_loop_on_sparse_tiles(ctx, dev, r, scheme, cover):
    import torch
    import ctdm_gb300 as C
    rng = np.random.default_rng([r, scheme, len(cover)])
    keep = voxels(r, cover, rng)
    accelerated, mode = cover in ("ends", "all"), int(cover in ("corner", "disc"))
    f = np.zeros((r, r, r))
    b = r // 8
    f[b:3 * b, 2 * b:5 * b, b:4 * b] = 0.05
    F2 = np.zeros((r, r, r), np.complex64)
    F2[keep] = (np.fft.fftn(-K2 * f) * (1 + 0.05 * rng.standard_normal((r, r, r))))[keep]
    F2[keep & ((F2.real == 0) | (F2.imag == 0))] += np.complex64(K2 * (1 + 1j))
    before = C.plans(r)[1], C.loop_scheme(r)
    if r == 256:
        C.set_loop_scheme(r, scheme)
    try:
        out = torch.empty((r, r, r), dtype=torch.complex64, device=dev)
        counts = torch.from_numpy(keep.astype(np.int32)).to(dev)
        ctx.positivity(torch.from_numpy(F2).to(dev), r, 3, K2, NM, out, mode, counts if mode else None,
                       accelerated=accelerated)
        torch.cuda.synchronize()
    finally:
        if r == 256:
            C.set_loop_scheme(r, before[1])
    ref = loop64(F2.astype(np.complex128), keep, 3, accelerated)
    assert np.sqrt(np.mean(np.abs(out.cpu().numpy() - ref) ** 2)) <= 1e-5
