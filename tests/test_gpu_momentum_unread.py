"""The accelerated loop's first iteration does not read the previous iterate, whatever an
earlier call left in its buffer: here NaN, which a read weighted by beta = 0 would send on.
(NaN data do not leave one, the projection clamps them; a k^2 beyond float does, since the
contrast is then n^2 * -inf + inf.)  Reference: the loop in float64 numpy, RMSE <= 1e-5."""
import numpy as np
import pytest

from test_gpu_active_tiles import K2, NM, loop64

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("r,scheme", [(128, 0), (256, 0), (256, 1), (256, 2), (384, 1)])
def test_first_iterate_is_not_read(ctx, dev, r, scheme):
    import torch
    import ctdm_gb300 as C
    with np.errstate(all="ignore"):
        k2 = np.float32(1e39)
        left = np.float32(NM) ** 2 * (-k2 / np.float32(NM) ** 2) + k2   # what the poisoned call keeps
        assert np.isnan(left) and np.isnan(np.float32(1) + np.float32(0) * (np.float32(1) - left))
    rng = np.random.default_rng([r, scheme])
    f = np.zeros((r, r, r))
    f[r // 8:r // 3, r // 4:r // 2, r // 8:r // 2] = 0.05
    F2 = np.fft.fftn(-K2 * f).astype(np.complex64)
    F2[(rng.random((r, r, r)) < 0.7) | (F2.real == 0) | (F2.imag == 0)] = 0
    before = C.loop_scheme(r)
    if r >= 256:
        C.set_loop_scheme(r, scheme)
    try:
        dF2 = torch.from_numpy(F2).to(dev)
        out = torch.empty_like(dF2)
        ctx.positivity(dF2, r, 2, 1e39, NM, out, accelerated=True)
        ctx.positivity(dF2, r, 2, K2, NM, out, accelerated=True)
        torch.cuda.synchronize()
    finally:
        if r >= 256:
            C.set_loop_scheme(r, before)
    ref = loop64(F2.astype(np.complex128), F2 != 0, 2, True)
    assert np.sqrt(np.mean(np.abs(out.cpu().numpy() - ref) ** 2)) <= 1e-5
