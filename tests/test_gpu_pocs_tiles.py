"""ASD-POCS on samples that cover few z tiles, at sides whose TV march takes fewer planes
per block than the reference workload's, against the FP64 oracle.  Tolerances as in the
line-scan tests: per-iteration distances 1e-3 relative, the output's RI RMSE <= 1e-5."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("r,cover", [(32, "ends"), (32, "dense"), (64, "half"), (128, "half")])
def test_pocs_on_sparse_tiles(ctx, dev, oracle, r, cover):
    import torch
    import ctdm_gb300 as C
    n_med, k2 = 1.337, 2.5e14
    rng = np.random.default_rng([r, len(cover)])
    s = np.fft.fftfreq(r, 1.0 / r)
    keep = np.zeros((r, r, r), bool)
    if cover == "dense":
        keep[rng.random((r, r, r)) < 0.4] = True
    elif cover == "half":
        keep[np.abs(s) < r / 5] = (np.hypot(s[:, None], s[None, :]) < r / 4)[None]
    else:
        keep[0, 0, 0] = keep[1, r - 1, 0] = keep[r - 1, 2, 7] = keep[3, r // 2, 8] = keep[2, 1, r - 1] = True
    z = np.linspace(-1, 1, r)
    v = 0.06 * (z[:, None, None] ** 2 + z[None, :, None] ** 2 + (z[None, None, :] - 0.1) ** 2 < 0.2)
    F2 = np.where(keep, -k2 * np.fft.fftn(v), 0).astype(np.complex64)
    F2[0, 0, 0] = np.complex64(F2[0, 0, 0].real)   # a sample with one zero part is measured
    op = oracle.pocs_params(iterations=3, tv_steps=4)
    ref, oh = oracle.pocs(F2.astype(np.complex128), op, k2, n_med)
    out = torch.zeros((r, r, r), dtype=torch.complex64, device=dev)
    h = ctx.pocs(torch.from_numpy(F2).to(dev), r, k2, n_med, out, params=C.pocs_params(iterations=3, tv_steps=4),
                 history=True)
    np.testing.assert_allclose(h, oh, rtol=1e-3, atol=1e-6)
    assert np.sqrt(np.mean(np.abs(out.cpu().numpy() - ref) ** 2)) <= 1e-5
