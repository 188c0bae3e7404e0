"""The DCT unwrap at every map side (one cluster launch up to 256, three launches above;
radix-3 sides, the twiddle quirk and the exact inverse), one map and several, against the
FP64 oracle.  Tolerance: the stage's phase bound, RMSE <= 1e-4 rad."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mode", [0, 1])
@pytest.mark.parametrize("m", [16, 32, 64, 128, 256, 384, 512, 768])
def test_every_side(ctx, dev, oracle, m, mode):
    import torch
    rng = np.random.default_rng([m, mode])
    maps = 3 if m <= 256 else 2
    yy, xx = np.mgrid[0:m, 0:m] / m
    p = np.stack([9 * np.sin(2.1 * xx + a) * np.cos(1.7 * yy) + 3 * xx for a in range(maps)])
    p += 0.02 * rng.standard_normal(p.shape)
    phi = (p - 2 * np.pi * np.round(p / (2 * np.pi))).astype(np.float32)
    d = torch.from_numpy(phi).to(dev)
    out = torch.empty_like(d)
    ctx.unwrap_dct(d, out, maps, m, mode)
    got = out.cpu().numpy()
    one = torch.empty_like(d[:1])
    ctx.unwrap_dct(d[1:2].contiguous(), one, 1, m, mode)
    assert np.array_equal(one.cpu().numpy()[0], got[1])
    for a in range(maps):
        assert np.sqrt(np.mean((got[a] - oracle.dct_unwrap(phi[a].astype(np.float64), mode)) ** 2)) <= 1e-4
