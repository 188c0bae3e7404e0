"""The accelerated loop's first and last iteration (no previous iterate read, none stored) on
the plane passes: one, two and three iterations, on a context whose last accelerated call
left NaN behind.  Reference: the loop in float64 numpy, RMSE <= 1e-5; one iteration is the
plain loop's to the bit."""
import numpy as np
import pytest

from test_gpu_active_tiles import K2, NM, loop64

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("iters", [1, 2, 3])
@pytest.mark.parametrize("r,scheme", [(128, 0), (256, 1), (256, 2), (384, 1)])
def test_momentum_ends(ctx, dev, r, scheme, iters):
    import torch
    import ctdm_gb300 as C
    rng = np.random.default_rng([r, scheme, iters])
    f = np.zeros((r, r, r))
    f[r // 8:r // 3, r // 4:r // 2, r // 8:r // 2] = 0.05
    F2 = np.fft.fftn(-K2 * f).astype(np.complex64)
    F2[(rng.random((r, r, r)) < 0.7) | (F2.real == 0) | (F2.imag == 0)] = 0
    keep = F2 != 0
    before = C.plans(r)[1], C.loop_scheme(r)
    if r >= 256:
        C.set_loop_scheme(r, scheme)
    try:
        dF2 = torch.from_numpy(F2).to(dev)
        out, plain = torch.empty_like(dF2), torch.empty_like(dF2)
        ctx.positivity(torch.full_like(dF2, float("nan")), r, 3, K2, NM, out, accelerated=True)
        ctx.positivity(dF2, r, iters, K2, NM, out, accelerated=True)
        ctx.positivity(dF2, r, iters, K2, NM, plain)
        torch.cuda.synchronize()
    finally:
        if r >= 256:
            C.set_loop_scheme(r, before[1])
    if iters == 1:
        assert torch.equal(out, plain)
    ref = loop64(F2.astype(np.complex128), keep, iters, True)
    assert np.sqrt(np.mean(np.abs(out.cpu().numpy() - ref) ** 2)) <= 1e-5
