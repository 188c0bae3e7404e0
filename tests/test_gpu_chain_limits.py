"""Around the sizes where a launch stops being chained to the one before it (clusters of the
DCT unwrap, the hologram row pass beyond one wave): calls in a row, many maps or frames
against one at a time, to the bit."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m,limit", [(64, 32), (128, 13), (256, 9)])
def test_unwrap(ctx, dev, m, limit):
    import torch
    g = torch.Generator(device=dev).manual_seed(m)
    phi = (torch.rand((limit + 1, m, m), generator=g, device=dev) - 0.5) * 6.2
    one, many = torch.empty_like(phi), torch.empty_like(phi)
    for a in range(limit + 1):
        ctx.unwrap_dct(phi[a:a + 1], one[a:a + 1], 1, m, 0)
    for maps in (limit, limit + 1, limit, limit + 1):
        many.zero_()
        ctx.unwrap_dct(phi, many, maps, m, 0)
        assert torch.equal(many[:maps], one[:maps])


@pytest.mark.parametrize("n,frames", [(256, 12), (512, 18), (512, 25)])
def test_hologram_rows(ctx, dev, n, frames):
    import torch
    g = torch.Generator(device=dev).manual_seed(n + frames)
    y, x = torch.meshgrid(torch.arange(n, device=dev), torch.arange(n, device=dev), indexing="ij")
    bg = (100 + 40 * torch.cos(2 * torch.pi * (0.31 * x + 0.22 * y))).float().contiguous()
    holo = (bg + 10 * torch.randn((frames, n, n), generator=g, device=dev)).contiguous()
    m = n // 4
    ph, am, p1, a1 = (torch.empty((frames, m, m), device=dev) for _ in range(4))
    for a in range(frames):
        ctx.qpi(n, m, holo[a:a + 1], bg, p1[a:a + 1], a1[a:a + 1], 1)
    for _ in range(3):
        ctx.qpi(n, m, holo, bg, ph, am, frames)
        assert torch.equal(ph, p1) and torch.equal(am, a1)
