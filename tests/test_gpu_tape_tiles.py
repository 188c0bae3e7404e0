"""The differentiable form on samples that cover few z tiles, and its TV gradient at the
edges of the 32 x 16 x planes march, against float64 numpy.  Tolerances: the operator's
and the gradient's relative L2 bound, 1e-5; the objective 1e-5 relative; contrasts after
three updates 1e-5 absolute RMS."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
K2 = 4.0


def tape64(r, keep, data, lam, eps):
    def fwd(v):
        return (np.fft.fftn(v) / r ** 1.5)[keep]

    def adj(y):
        w = np.zeros((r, r, r), np.complex128)
        w[keep] = y
        return np.fft.ifftn(w) * r ** 1.5

    def obj(v):
        res = fwd(v) - data
        g, loss = adj(res), 0.5 * np.sum(np.abs(res) ** 2)
        if lam:
            d = [np.concatenate([np.diff(v, axis=a), np.zeros_like(np.take(v, [0], a))], a) for a in range(3)]
            mag = np.sqrt(sum(np.abs(e) ** 2 for e in d) + eps * eps)
            loss += lam * mag.sum()
            for a, e in enumerate(d):
                q = e / mag
                g -= lam * q
                sl, sr = [slice(None)] * 3, [slice(None)] * 3
                sl[a], sr[a] = slice(1, None), slice(None, -1)
                g[tuple(sl)] += lam * q[tuple(sr)]
        return loss, g
    return fwd, adj, obj


@pytest.mark.parametrize("r", [32, 64, 128])
@pytest.mark.parametrize("cover", ["one", "ends", "column", "dense"])
def test_tape_on_sparse_tiles(ctx, dev, r, cover):
    import torch
    import ctdm_gb300 as C
    rng = np.random.default_rng([r, len(cover)])
    keep = np.zeros((r, r, r), bool)
    if cover == "one":
        keep[r - 1, r - 1, r - 1] = True
    elif cover == "ends":
        keep[0, 0, 0] = keep[3, 1, r - 1] = keep[5, r - 1, 8] = keep[6, r // 2, 7] = True
    elif cover == "column":
        keep[:, 2, 9] = True
    else:
        keep[rng.random((r, r, r)) < 0.3] = True
    lam, eps, positive = (0.0 if cover == "ends" else 0.02), 1e-2, cover in ("one", "dense")
    F2 = np.where(keep, rng.standard_normal((r, r, r)) + 1j * rng.standard_normal((r, r, r)), 0).astype(np.complex64)
    F2 *= np.float32(-K2 * r ** 1.5 * 0.1)
    V = (0.1 * (rng.standard_normal((r, r, r)) + 1j * rng.standard_normal((r, r, r)))).astype(np.complex64)
    dt = lambda a: torch.from_numpy(np.ascontiguousarray(a)).to(dev)   # noqa: E731
    tape = C.Tape(dt(F2), r, K2, dt(keep.astype(np.int32)))
    data = F2.astype(np.complex128)[keep] / (-K2 * r ** 1.5)
    fwd, adj, obj = tape64(r, keep, data, lam, eps)
    rel = lambda a, b: np.linalg.norm(a - b) / np.linalg.norm(b)       # noqa: E731
    y = torch.empty(tape.samples, dtype=torch.complex64, device=dev)
    g = torch.full((r, r, r), float("nan"), dtype=torch.complex64, device=dev)
    tape.forward(dt(V), y)
    assert rel(y.cpu().numpy(), fwd(V)) < 1e-5
    tape.backward(y, g)
    assert rel(g.cpu().numpy(), adj(y.cpu().numpy().astype(np.complex128))) < 1e-5
    g.fill_(float("nan"))
    loss = tape.loss_grad(dt(V), g, lam, eps)
    l64, g64 = obj(V.astype(np.complex128))
    assert abs(loss - l64) <= 1e-5 * l64 and rel(g.cpu().numpy(), g64) < 1e-5
    W, x, t = V.astype(np.complex128), V.astype(np.complex128), 1.0
    tau = 1.0 / (1.0 + 12.0 * lam / eps)
    for _ in range(3):
        xn = W - tau * obj(W)[1]
        if positive:
            s = np.sqrt(1 + xn)
            xn = (np.maximum(s.real, 1) + 1j * np.maximum(s.imag, 0)) ** 2 - 1
        tn = 0.5 * (1 + np.sqrt(1 + 4 * t * t))
        W, x, t = xn + (t - 1) / tn * (xn - x), xn, tn
    v = dt(V)
    tape.reconstruct(v, 3, lam, eps, positivity=positive)
    assert np.sqrt(np.mean(np.abs(v.cpu().numpy() - x) ** 2)) <= 1e-5
    tape.close()
