"""Timing cases: what users of this framework have it do, over the range of sizes and options they use.

A case is a dict of plain values.  `prepare` makes what a program holds before the call (device
or pinned host inputs, the parameters, the kept context), `run` is one pass through the public
entry points, `exact` the same mathematics in 64 bits with torch alone.

Inputs are synthetic acquisitions: ellipsoid specimens, first-order Rytov fields on the Ewald
caps, off-axis holograms with shot noise, wrapped phase maps, and measured k-space volumes.
"""
import math

import numpy as np
import torch

import ctdm_gb300 as C

DEV = "cuda:0"
WAVELENGTH, N_MED, NA = 532e-9, 1.337, 0.9
F64, C128 = torch.float64, torch.complex128
_CONTEXT = []


def _context():
    """The device context a program creates once and keeps (workspace, tables)."""
    if not _CONTEXT:
        _CONTEXT.append(C.Context(0))
    return _CONTEXT[0]


# ---------------------------------------------------------------- cases
def listed():
    return [
        # the headline acquisition: 121 angles of a thick specimen, both unwrappers, 20 loop bodies
        dict(name="tomogram_wrap_heavy", kind="tomogram", angles=121, n=1024, r=256, pixel=1e-7, iterations=20,
             goldstein=True, accelerated=False, mask=False, dn=0.063, counts=0),
        # live preview: a few 8-bit camera frames from host memory, a small volume back to the host
        dict(name="preview_u8", kind="tomogram", angles=16, n=256, r=64, pixel=4e-7, iterations=5, goldstein=False,
             accelerated=False, mask=False, dn=0.02, counts=1),
        # phase retrieval alone (quantitative phase imaging of a thin specimen), 2-D window
        dict(name="qpi_a_1024", kind="qpi", method="a", angles=31, n=1024),
        # the reference's default phase retrieval (1-D filter), ordinary frames
        dict(name="qpi_b_512", kind="qpi", method="b", angles=49, n=512),
        # one small map while the specimen is being focused: the smallest call
        dict(name="unwrap_one_128", kind="unwrap", maps=1, m=128, mode=1),
        # the maps of a whole scan, the reference's inverse twiddle
        dict(name="unwrap_scan_256", kind="unwrap", maps=121, m=256, mode=0),
        # branch cuts of a scan of noisy maps
        dict(name="goldstein_256", kind="goldstein", maps=49, w=256, h=256, noise=0.35),
        # per-angle spectra and Fourier mapping of a large scan
        dict(name="mapping_512", kind="mapping", angles=181, m=256, n=1024, r=512, pixel=1e-7),
        # the constrained loop on a mid-size volume, hit-mask replacement
        dict(name="loop_mask_384", kind="loop", angles=121, r=384, pixel=1e-7, iterations=10, mask=True,
             accelerated=False),
        # the accelerated loop on a large volume: the largest call
        dict(name="loop_accel_512", kind="loop", angles=181, r=512, pixel=1e-7, iterations=10, mask=False,
             accelerated=True),
        # the differentiable form: operator, adjoint, objective gradient, regularised descent
        dict(name="gradient_256", kind="gradient", angles=121, r=256, pixel=1e-7, iterations=4, lam=1e-3,
             positivity=True),
        # total-variation POCS on a one-axis scan
        dict(name="pocs_256", kind="pocs", angles=121, r=256, pixel=1e-7, iterations=3, tv_steps=20),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _pixel(r):
    """Voxels of the acquisitions in use: 0.1 um at full size, coarser for small volumes."""
    return 4e-7 if r <= 64 else 2e-7 if r == 128 else 1e-7


def draw(rng):
    kind = rng.choice(["tomogram", "tomogram", "qpi", "unwrap", "goldstein", "mapping", "loop", "loop", "gradient",
                       "pocs"])
    if kind == "tomogram":
        n, r = rng.choice([(128, 32), (256, 64), (256, 128), (256, 256), (512, 256), (512, 384), (1024, 256)])
        return dict(kind=kind, angles=_log(rng, 8, 121), n=n, r=r, pixel=_pixel(r), iterations=rng.randint(1, 20),
                    goldstein=rng.random() < 0.3, accelerated=rng.random() < 0.3, mask=rng.random() < 0.3,
                    dn=rng.uniform(0.01, 0.06), counts=rng.choice([0, 0, 1, 2, 4]))
    if kind == "qpi":
        return dict(kind=kind, method=rng.choice(["a", "a", "b"]), angles=_log(rng, 1, 61),
                    n=rng.choice([256, 512, 1024, 2048]))
    if kind == "unwrap":
        return dict(kind=kind, maps=_log(rng, 1, 181), m=rng.choice([64, 128, 256, 384, 512]), mode=rng.randint(0, 1))
    if kind == "goldstein":
        return dict(kind=kind, maps=_log(rng, 1, 121), w=_log(rng, 48, 256), h=_log(rng, 48, 256),
                    noise=rng.uniform(0.1, 0.4))
    if kind == "mapping":
        n, r = rng.choice([(256, 64), (256, 128), (256, 256), (512, 256), (1024, 256), (512, 384), (1024, 512)])
        return dict(kind=kind, angles=_log(rng, 9, 181), m=n // 4, n=n, r=r, pixel=_pixel(r))
    r = rng.choice([64, 128, 256, 256, 384])
    if kind == "loop":
        return dict(kind=kind, angles=_log(rng, 16, 181), r=r, pixel=_pixel(r), iterations=rng.randint(1, 20),
                    mask=rng.random() < 0.4, accelerated=rng.random() < 0.4)
    if kind == "gradient":
        return dict(kind=kind, angles=_log(rng, 16, 121), r=r, pixel=_pixel(r), iterations=rng.randint(1, 3),
                    lam=rng.choice([0.0, 1e-4, 1e-3]), positivity=rng.random() < 0.5)
    return dict(kind="pocs", angles=_log(rng, 16, 121), r=r, pixel=_pixel(r), iterations=rng.randint(1, 2),
                tv_steps=rng.randint(5, 20))


# ---------------------------------------------------------------- synthetic data
def _generator(seed):
    g = torch.Generator(device=DEV)
    g.manual_seed(int(seed) * 7919 + 17)
    return g


def _specimen(seed, fov, dn):
    """A cell and a few denser bodies inside it: (centre, semi-axes, index step) in metres."""
    rng = np.random.default_rng([int(seed), 5])
    cell = np.array([rng.uniform(0.16, 0.2), rng.uniform(0.13, 0.17), rng.uniform(0.11, 0.14)]) * fov
    cell = np.minimum(cell, 5e-6)
    parts = [(np.zeros(3), cell, dn)]
    for _ in range(3):
        r = rng.uniform(0.15, 0.3) * cell.min()
        parts.append((rng.uniform(-0.4, 0.4, 3) * cell, np.full(3, r), 0.3 * dn * rng.uniform(0.5, 1.0)))
    return parts


def _potential(parts, kx, ky, kz):
    """Fourier transform of the scattering potential at the given frequencies (1/m)."""
    k0 = 2 * math.pi / WAVELENGTH
    out = torch.zeros(kx.shape, dtype=C128, device=DEV)
    for c, s, dn in parts:
        q = 2 * math.pi * torch.sqrt((s[0] * kx) ** 2 + (s[1] * ky) ** 2 + (s[2] * kz) ** 2)
        q = torch.clamp(q, min=1e-3)
        shape = 3.0 * (torch.sin(q) - q * torch.cos(q)) / q ** 3
        step = -k0 * k0 * ((N_MED + dn) ** 2 - N_MED ** 2) * 4.0 / 3.0 * math.pi * float(np.prod(s))
        arg = -2 * math.pi * (kx * c[0] + ky * c[1] + kz * c[2])
        out += step * shape * torch.exp(torch.complex(torch.zeros_like(arg), arg))
    return out


def _angles(count, scan="cone"):
    if scan == "line":
        t = math.asin(NA / N_MED)
        return np.linspace(-t, t, count).astype(np.float32), np.zeros(count, np.float32)
    phi = 2 * np.pi * np.arange(count) / count
    s = NA / N_MED
    return np.arcsin(s * np.sin(phi)).astype(np.float32), np.arcsin(s * np.cos(phi)).astype(np.float32)


def _signed(n):
    return torch.fft.fftfreq(n, 1.0 / n, dtype=F64, device=DEV)


def _holograms(seed, angles, n, pixel, dn, photons, carrier, levels):
    """Sample holograms (angles, n, n), the background (n, n) and the angles."""
    g = _generator(seed)
    ax, ay = _angles(angles)
    parts = _specimen(seed, n * pixel, dn)
    fm0, df = N_MED / WAVELENGTH, 1.0 / (n * pixel)
    sgn = _signed(n) * df
    yy, xx = torch.meshgrid(torch.arange(n, dtype=F64, device=DEV), torch.arange(n, dtype=F64, device=DEV),
                            indexing="ij")
    arg = -2 * math.pi * (carrier[0] * xx + carrier[1] * yy)
    ref = torch.complex(torch.cos(arg), torch.sin(arg))
    holo = torch.empty((angles, n, n), dtype=torch.float32, device=DEV)
    for a in range(angles):
        fx0, fy0 = fm0 * math.sin(float(ay[a])), fm0 * math.sin(float(ax[a]))
        fz0 = math.sqrt(fm0 * fm0 - fx0 * fx0 - fy0 * fy0)
        rad = fm0 * fm0 - ((sgn + fx0) ** 2)[None, :] - ((sgn + fy0) ** 2)[:, None]
        iy, ix = torch.nonzero(rad > (0.02 * fm0) ** 2, as_tuple=True)
        fz = torch.sqrt(rad[iy, ix])
        spec = torch.zeros((n, n), dtype=C128, device=DEV)
        spec[iy, ix] = _potential(parts, sgn[ix], sgn[iy], fz - fz0) / (4j * math.pi * fz) / (pixel * pixel)
        u = torch.fft.fftshift(torch.fft.ifft2(spec)).T
        holo[a] = torch.poisson((photons / 2 * (ref + torch.exp(u)).abs() ** 2).float(), generator=g)
    bg = torch.poisson((photons / 2 * (ref + 1.0).abs() ** 2).float(), generator=g)
    if levels:
        holo.clamp_(max=levels)
        bg.clamp_(max=levels)
    return holo, bg, ax, ay


def _tomogram_data(case, seed):
    photons, levels = {0: (1000.0, 0), 4: (1000.0, 0), 2: (1000.0, 65535), 1: (60.0, 255)}[case["counts"]]
    return _holograms(seed, case["angles"], case["n"], case["pixel"], case["dn"], photons, (0.125, 0.125), levels)


def _qpi_data(case, seed):
    carrier = (0.125, 0.125) if case["method"] == "a" else (0.25, 0.0)
    return _holograms(seed, case["angles"], case["n"], 1e-7, 0.01, 1000.0, carrier, 0)


def _smooth(seed, maps, h, w, peak, noise):
    """True phase of `maps` views of a specimen (rad), with phase noise."""
    g = _generator(seed)
    yy = torch.linspace(-1, 1, h, device=DEV)[None, :, None]
    xx = torch.linspace(-1, 1, w, device=DEV)[None, None, :]
    u = torch.rand((5, maps, 1, 1), generator=g, device=DEV) * 2 - 1
    phase = peak * torch.clamp(1 - ((xx - 0.2 * u[0]) / 0.6) ** 2 - ((yy - 0.2 * u[1]) / 0.5) ** 2, min=0.0)
    phase += 0.2 * peak * torch.exp(-((xx - 0.3 * u[2]) ** 2 + (yy - 0.3 * u[3]) ** 2) / 0.02) + 0.5 * u[4] * xx
    return phase + noise * torch.randn((maps, h, w), generator=g, device=DEV)


def _wrapped(seed, maps, h, w, peak, noise):
    p = _smooth(seed, maps, h, w, peak, noise).double()
    return (p - 2 * math.pi * torch.round(p / (2 * math.pi))).float().contiguous()


def _maps(case, seed):
    """Unwrapped phase and amplitude maps of a scan."""
    m, a = case["m"], case["angles"]
    phase = _smooth(seed, a, m, m, 4.0, 0.02).float().contiguous()
    amp = torch.exp(0.1 * _smooth(seed + 1000003, a, m, m, -2.0, 0.1)).float().contiguous()
    return phase, amp


def _cap(ax, ay, a, fm0, df, r):
    """Voxel z index of each detector frequency of angle a, where it has one, and f_z."""
    fx0, fy0 = fm0 * math.sin(float(ay[a])), fm0 * math.sin(float(ax[a]))
    rad0 = fm0 * fm0 - fx0 * fx0 - fy0 * fy0
    sgn = _signed(r)
    fx, fy = sgn * df + fx0, sgn * df + fy0
    rad = fm0 * fm0 - ((fx * fx)[None, :] + (fy * fy)[:, None])
    fz = torch.sqrt(torch.clamp(rad, min=0.0))
    t = (fz - math.sqrt(max(rad0, 0.0))) / df
    nz = torch.where(t > 0, torch.floor(t + 0.5), torch.ceil(t - 0.5)).long() % r
    return (rad >= 0) & (rad0 >= 0), nz, fz


def _geometry(case):
    fm0, dx, r = N_MED / WAVELENGTH, case["pixel"], case["r"]
    k = 2 * math.pi * N_MED / WAVELENGTH
    return fm0, 1.0 / (r * dx), dx, k * k


def _kspace(case, seed, scan="cone"):
    """Measured volume F2 (zero where nothing was measured) and the hit counts, [z][y][x]."""
    r = case["r"]
    fm0, df, dx, _ = _geometry(case)
    ax, ay = _angles(case["angles"], scan)
    counts = torch.zeros(r * r * r, dtype=torch.int32, device=DEV)
    plane = torch.arange(r * r, device=DEV).reshape(r, r)
    for a in range(case["angles"]):
        ok, nz, _ = _cap(ax, ay, a, fm0, df, r)
        counts[(nz * r * r + plane)[ok]] += 1
    at = torch.nonzero(counts, as_tuple=True)[0]
    sgn = _signed(r) * df
    vals = _potential(_specimen(seed, r * dx, 0.04), sgn[at % r], sgn[(at // r) % r], sgn[at // (r * r)]) / dx ** 3
    noise = torch.randn((2, at.numel()), generator=_generator(seed), device=DEV, dtype=F64)
    vals += 0.02 * vals.abs().square().mean().sqrt() * torch.complex(noise[0], noise[1])
    f2 = torch.zeros(r * r * r, dtype=torch.complex64, device=DEV)
    f2[at] = vals.to(torch.complex64)
    return f2.reshape(r, r, r), counts.reshape(r, r, r)


# ---------------------------------------------------------------- prepare and run
def _volume(r):
    return torch.empty((r, r, r), dtype=torch.complex64, device=DEV)


def prepare(case, seed):
    kind = case["kind"]
    s = dict(case=case, ctx=_context())
    if kind == "tomogram":
        holo, bg, ax, ay = _tomogram_data(case, seed)
        s["params"] = C.default_params(n_holo=case["n"], r_vol=case["r"], iterations=case["iterations"], n_med=N_MED,
                                       wavelength=WAVELENGTH, dx=case["pixel"], run_goldstein=int(case["goldstein"]),
                                       accelerated=int(case["accelerated"]), check_mode=int(case["mask"]))
        out = torch.empty((case["r"],) * 3, dtype=torch.complex64, device=DEV)
        if case["counts"]:   # host call: camera counts or floats in pinned memory
            t = {1: torch.uint8, 2: torch.uint16, 4: torch.float32}[case["counts"]]
            holo, bg = (x.to(t).cpu().pin_memory().numpy() for x in (holo, bg))
            out = torch.empty((case["r"],) * 3, dtype=torch.complex64).pin_memory().numpy()
        s.update(holo=holo, bg=bg, ax=ax, ay=ay, out=out)
    elif kind == "qpi":
        s["holo"], s["bg"], _, _ = _qpi_data(case, seed)
        s["phase"], s["amp"] = (torch.empty((case["angles"], case["n"] // 4, case["n"] // 4), device=DEV)
                                for _ in range(2))
    elif kind == "unwrap":
        s["phi"] = _wrapped(seed, case["maps"], case["m"], case["m"], 12.0, 0.05)
        s["out"] = torch.empty_like(s["phi"])
    elif kind == "goldstein":
        s["phi"] = _wrapped(seed, case["maps"], case["h"], case["w"], 8.0, case["noise"])
        s["charges"] = torch.empty(s["phi"].shape, dtype=torch.int8, device=DEV)
        s["cuts"] = torch.empty(s["phi"].shape, dtype=torch.uint8, device=DEV)
        s["out"] = torch.empty_like(s["phi"])
    elif kind == "mapping":
        s["phase"], s["amp"] = _maps(case, seed)
        s["ax"], s["ay"] = _angles(case["angles"])
        r = case["r"]
        s["u"] = torch.empty((case["angles"], r, r), dtype=torch.complex64, device=DEV)
        s["f2"], s["counts"] = _volume(r), torch.empty((r, r, r), dtype=torch.int32, device=DEV)
    elif kind == "loop":
        s["f2"], s["counts"] = _kspace(case, seed)
        s["out"] = _volume(case["r"])
    elif kind == "gradient":
        s["f2"], counts = _kspace(case, seed)
        s["tape"] = C.Tape(s["f2"], case["r"], _geometry(case)[3], counts)
        n = s["tape"].samples
        s["v0"] = _contrast(case, seed)
        s["v"], s["adj"], s["grad"] = _volume(case["r"]), _volume(case["r"]), _volume(case["r"])
        s["y"] = torch.empty(n, dtype=torch.complex64, device=DEV)
    else:
        s["f2"], _ = _kspace(case, seed, "line")
        s["out"] = _volume(case["r"])
        s["pocs"] = C.pocs_params(iterations=case["iterations"], tv_steps=case["tv_steps"])
    return s


def _contrast(case, seed):
    """A starting contrast: a soft ball with a little noise."""
    r = case["r"]
    z = torch.linspace(-1, 1, r, device=DEV)
    d = z[:, None, None] ** 2 + z[None, :, None] ** 2 + z[None, None, :] ** 2
    noise = torch.randn((2, r, r, r), generator=_generator(seed + 31), device=DEV) * 1e-3
    return torch.complex(0.05 * torch.exp(-d / 0.1) + noise[0], noise[1]).contiguous()


def run(s):
    case, ctx = s["case"], s["ctx"]
    kind = case["kind"]
    if kind == "tomogram":
        if case["counts"]:
            return ctx.reconstruct(s["params"], s["holo"], s["bg"], s["ax"], s["ay"], s["out"])
        ctx.reconstruct_device(s["params"], s["holo"], s["bg"], s["ax"], s["ay"], s["out"])
        return s["out"]
    if kind == "qpi":
        if case["method"] == "a":
            ctx.qpi(case["n"], case["n"] // 4, s["holo"], s["bg"], s["phase"], s["amp"], case["angles"])
        else:
            ctx.qpi_b(case["n"], s["holo"], s["bg"], s["phase"], s["amp"], case["angles"])
        return s["phase"], s["amp"]
    if kind == "unwrap":
        ctx.unwrap_dct(s["phi"], s["out"], case["maps"], case["m"], case["mode"])
        return s["out"]
    if kind == "goldstein":
        ctx.goldstein(s["phi"], s["charges"], s["cuts"], s["out"], case["maps"], case["w"], case["h"])
        return s["charges"], s["cuts"], s["out"]
    fm0, df, dx, k2 = _geometry(case)
    if kind == "mapping":
        ctx.prepare_spectra(s["phase"], s["amp"], s["u"], case["angles"], case["m"], case["n"], case["r"])
        ctx.map_ewald(s["u"], s["ax"], s["ay"], fm0, df, dx, s["f2"], s["counts"])
        return s["u"], s["f2"], s["counts"]
    if kind == "loop":
        ctx.positivity(s["f2"], case["r"], case["iterations"], k2, N_MED, s["out"], int(case["mask"]),
                       s["counts"] if case["mask"] else None, accelerated=case["accelerated"])
        return s["out"]
    if kind == "gradient":
        tape = s["tape"]
        tape.forward(s["v0"], s["y"])
        tape.backward(s["y"], s["adj"])
        loss = tape.loss_grad(s["v0"], s["grad"], case["lam"])
        s["v"].copy_(s["v0"])
        tape.reconstruct(s["v"], case["iterations"], case["lam"], positivity=case["positivity"])
        return dict(y=s["y"], adjoint=s["adj"], loss=loss, grad=s["grad"], v=s["v"])
    ctx.pocs(s["f2"], case["r"], k2, N_MED, s["out"], s["pocs"])
    return s["out"]


# ---------------------------------------------------------------- work
def _fft_flops(points, length):
    return 5.0 * points * math.log2(length)


def work(case):
    kind = case["kind"]
    if kind in ("tomogram", "qpi"):
        a, n = case["angles"], case["n"]
        m = n // 4
        by = a * n * n * (case.get("counts") or 4) + n * n * 4
        fl = a * (_fft_flops(n * n, n * n) / 2 + 2 * _fft_flops(m * m, m * m))
        if kind == "qpi":
            return dict(bytes=by + a * m * m * 8, flops=fl)
        r3 = case["r"] ** 3
        fl += a * _fft_flops(case["r"] ** 2, case["r"] ** 2) + 2 * a * _fft_flops(m * m, m * m)
        return dict(bytes=by + r3 * 8, flops=fl + (2 * case["iterations"] + 1) * _fft_flops(r3, r3))
    if kind == "unwrap":
        p = case["maps"] * case["m"] ** 2
        return dict(bytes=8 * p, flops=2 * _fft_flops(p, case["m"] ** 2))
    if kind == "goldstein":
        p = case["maps"] * case["w"] * case["h"]
        return dict(bytes=10 * p, flops=40 * p)
    r = case["r"]
    r2, r3 = r * r, r ** 3
    if kind == "mapping":
        a = case["angles"]
        return dict(bytes=8 * a * case["m"] ** 2 + 16 * a * r2 + 12 * r3, flops=a * _fft_flops(r2, r2) + 40 * a * r2)
    if kind == "loop":
        return dict(bytes=r3 * (20 if case["mask"] else 16), flops=(2 * case["iterations"] + 1) * _fft_flops(r3, r3))
    if kind == "gradient":
        return dict(bytes=40 * r3, flops=(4 + 2 * case["iterations"]) * (_fft_flops(r3, r3) + 20 * r3))
    return dict(bytes=16 * r3, flops=case["iterations"] * (2 * _fft_flops(r3, r3) + 25 * r3 * case["tv_steps"]))


# ---------------------------------------------------------------- the same in 64 bits
def _exact_window(x, r0, c0, rad, n, m):
    """Window of the spectrum around the carrier, masked and swapped, back to the image plane."""
    j = torch.arange(m, device=DEV) - m // 2
    w = torch.fft.fft2(x.double())[..., (r0 - n // 2 + j) % n, :][..., (c0 - n // 2 + j) % n]
    keep = j.abs() <= rad
    w = w * (keep[:, None] & keep[None, :])
    return torch.fft.ifft2(torch.fft.ifftshift(w, dim=(-2, -1))).conj()


def _phase_amp(v, g):
    return torch.angle(g) - torch.angle(v), v.abs() / g.abs()


def _exact_qpi_a(holo, bg, n):
    m = n // 4
    mag = torch.fft.fftshift(torch.fft.fft2(bg.double()).abs())
    start = 600 * n // 1024
    at = int(torch.argmax(mag[start:].reshape(-1)))
    r0, c0 = start + at // n, at % n
    rad = abs(r0 - n // 2) // 3
    g = _exact_window(bg, r0, c0, rad, n, m)
    pairs = [_phase_amp(_exact_window(h, r0, c0, rad, n, m), g) for h in holo]
    return torch.stack([p for p, _ in pairs]), torch.stack([a for _, a in pairs])


def _bilinear(img, rows, cols, ry, rx):
    """Bilinear taps at (rows ry, cols rx); taps past the edge read 0."""
    h, w = img.shape[-2:]
    p = torch.nn.functional.pad(img, (0, 2, 0, 2))
    y, x = rows * ry, cols * rx
    iy, ix = torch.floor(y).long(), torch.floor(x).long()
    a, b = (x - ix)[None, :], (y - iy)[:, None]
    iy, ix = iy.clamp(max=h), ix.clamp(max=w)
    d00, d10 = p[..., iy[:, None], ix[None, :]], p[..., iy[:, None], ix[None, :] + 1]
    d01, d11 = p[..., iy[:, None] + 1, ix[None, :]], p[..., iy[:, None] + 1, ix[None, :] + 1]
    return (1 - b) * ((1 - a) * d00 + a * d10) + b * ((1 - a) * d01 + a * d11)


def _exact_qpi_b(holo, bg, n):
    m = n // 4
    rows, cols = torch.arange(m, dtype=F64, device=DEV), torch.arange(n, dtype=F64, device=DEV)
    xr, yr = float(np.float32(n - 1) / np.float32(n)), float(np.float32(n - 1) / np.float32(m))

    def spectrum(h):
        return torch.fft.fftshift(torch.fft.fft(_bilinear(h.double(), rows, cols, yr, xr), dim=-1), dim=-1)

    def centre(sp):
        lo = int(n * 0.6)
        c = lo + int(torch.argmax(sp.abs().sum(dim=0)[lo:]))
        return n - c if n - c < m // 2 else c

    def field(sp, c):
        k = torch.arange(m, device=DEV) - n // 8 + c
        ok = (k >= 0) & (k < n)
        w = sp[:, k.clamp(0, n - 1)] * ok
        return torch.fft.ifft(torch.fft.ifftshift(w, dim=-1), dim=-1).conj().T

    sb = spectrum(bg)
    cb = centre(sb)
    g = field(sb, cb)
    out = []
    for a, h in enumerate(holo):
        sp = spectrum(h)
        out.append(_phase_amp(field(sp, centre(sp) if a == 0 else cb), g))
    return torch.stack([p for p, _ in out]), torch.stack([q for _, q in out])


def _exact_unwrap(phi, mode):
    m = phi.shape[-1]

    def wrap(t):   # differences as the single-precision maps give them
        t = t.double()
        return t - 2 * math.pi * torch.sign(t) * torch.floor((math.pi * torch.sign(t) + t).abs() / (2 * math.pi))

    gx, gy = (torch.zeros(phi.shape, dtype=F64, device=DEV) for _ in range(2))
    gx[..., :-1] = wrap(phi[..., 1:] - phi[..., :-1])
    gy[..., :-1, :] = wrap(phi[..., 1:, :] - phi[..., :-1, :])
    lap = gx + gy
    lap[..., 1:] -= gx[..., :-1]
    lap[..., 1:, :] -= gy[..., :-1, :]
    k = torch.arange(m, dtype=F64, device=DEV)
    th = k * math.pi / (2 * m)
    tw = torch.complex(torch.cos(th), torch.sin(th))
    d_t = 1.0 / math.sqrt(2.0 * m)
    scale = torch.full((m,), d_t, dtype=F64, device=DEV)
    scale[0] /= math.sqrt(2.0)

    def dct(x):
        return (torch.fft.fft(torch.cat([x, x.flip(-1)], dim=-1))[..., :m] * tw.conj()).real * scale

    def idct(x):
        first = x * d_t * tw
        first[..., 0] *= math.sqrt(2.0)
        i = torch.arange(1, m, device=DEV)
        t2 = (i + 1 if mode == 0 else i).double() * math.pi / (2 * m)
        second = -1j * torch.complex(torch.cos(t2), torch.sin(t2)) * x[..., m - i] * d_t
        v = torch.cat([first, torch.zeros_like(first[..., :1]), second], dim=-1)
        return (torch.fft.ifft(v) * (2 * m)).real[..., :m]

    e = 4 * torch.sin(2 * math.pi * k / (4 * m - 1)) ** 2
    den = -(e[:, None] + e[None, :])
    den[0, 0] = 1.0
    x = dct(dct(lap).transpose(-1, -2)).transpose(-1, -2) / den
    x[..., 0, 0] = 0.0
    return idct(idct(x.transpose(-1, -2)).transpose(-1, -2))


def _exact_spectra(phase, amp, m, n, r):
    idx = torch.arange(r, dtype=F64, device=DEV) + (n - r) // 2
    ratio = float(np.float32(m - 1) / np.float32(n))

    def median(x):
        w = x.unfold(-2, 3, 1).unfold(-2, 3, 1).reshape(r - 2, r - 2, 9)
        y = x.clone()
        y[1:-1, 1:-1] = w.median(dim=-1).values
        return y

    out = []
    for p, a in zip(phase, amp):
        p, a = (_bilinear(v.double(), idx, idx, ratio, ratio) for v in (p, a))
        p, a = median(torch.where(torch.isfinite(p), p, 0.0)), median(torch.where(torch.isfinite(a), a, 1.0))
        a = torch.where(a == 0, 0.01, a.abs())
        u = torch.complex(torch.log(a), p).T
        out.append(torch.fft.fft2(torch.roll(u, (r // 2, r // 2), (0, 1))))
    return torch.stack(out)


def _exact_mapping(u, ax, ay, fm0, df, dx):
    r = u.shape[-1]
    f = torch.zeros(r * r * r, dtype=C128, device=DEV)
    cnt = torch.zeros(r * r * r, dtype=F64, device=DEV)
    plane = torch.arange(r * r, device=DEV).reshape(r, r)
    for a in range(u.shape[0]):
        ok, nz, fz = _cap(ax, ay, a, fm0, df, r)
        at = (nz * r * r + plane)[ok]
        f[at] += (4j * math.pi * fz * u[a])[ok]
        cnt[at] += 1
    f /= cnt.clamp(min=1.0)
    return (f / float(np.float32(dx))).reshape(r, r, r), cnt.reshape(r, r, r)


def _index(v, n_med):
    """n = n_med sqrt(1 + v), Re n >= n_med and Im n >= 0."""
    n = n_med * torch.sqrt(1.0 + v)
    return torch.complex(n.real.clamp(min=n_med), n.imag.clamp(min=0.0))


def _exact_loop(f2, keep, iterations, k2, accelerated):
    n_med = float(np.float32(N_MED))
    v = torch.fft.ifftn(f2) / -k2
    data = (f2 / -k2)[keep]
    prev, t = None, 1.0
    for _ in range(iterations):
        x = (_index(v, n_med) / n_med) ** 2 - 1.0
        tn = 0.5 * (1 + math.sqrt(1 + 4 * t * t))
        v = x + (t - 1) / tn * (x - prev) if accelerated and prev is not None else x
        prev, t = (x if accelerated else None), tn
        v = torch.fft.fftn(v)
        v[keep] = data
        v = torch.fft.ifftn(v)
    return torch.roll(_index(v, n_med), (f2.shape[0] // 2,) * 3, (0, 1, 2))


def _exact_gradient(case, seed):
    r, lam, eps = case["r"], case["lam"], 1e-4
    f2, counts = _kspace(case, seed)
    v0 = _contrast(case, seed).to(C128)
    keep = counts > 0
    unit = r ** 1.5
    data = f2.to(C128)[keep] / (-_geometry(case)[3] * unit)

    def forward(v):
        return (torch.fft.fftn(v) / unit)[keep]

    def backward(y):
        w = torch.zeros((r, r, r), dtype=C128, device=DEV)
        w[keep] = y
        return torch.fft.ifftn(w) * unit

    def tv(v):
        d = []
        for ax in range(3):
            e = torch.zeros_like(v)
            e.narrow(ax, 0, r - 1).copy_(v.narrow(ax, 1, r - 1) - v.narrow(ax, 0, r - 1))
            d.append(e)
        mag = torch.sqrt(sum(e.abs() ** 2 for e in d) + eps * eps)
        g = torch.zeros_like(v)
        for ax, e in enumerate(d):
            q = e / mag
            g -= q
            g.narrow(ax, 1, r - 1).add_(q.narrow(ax, 0, r - 1))
        return float(mag.sum()), g

    def gradient(v):
        res = forward(v) - data
        g = backward(res)
        loss = 0.5 * float(res.abs().square().sum())
        if lam:
            t, tg = tv(v)
            loss, g = loss + lam * t, g + lam * tg
        return loss, g

    y = forward(v0)
    loss, grad = gradient(v0)
    v, w, t = v0.clone(), v0.clone(), 1.0
    tau = 1.0 / (1.0 + 12.0 * lam / eps)
    for _ in range(case["iterations"]):
        x = w - tau * gradient(w)[1]
        if case["positivity"]:
            x = _index(x, 1.0) ** 2 - 1.0
        tn = 0.5 * (1 + math.sqrt(1 + 4 * t * t))
        w, v, t = x + (t - 1) / tn * (x - v), x, tn
    return dict(y=y, adjoint=backward(y), loss=loss, grad=grad, v=v)


def _exact_pocs(f2, k2, case):
    n_med, eps = float(np.float32(N_MED)), float(np.float32(1e-8))
    keep = f2 != 0
    data = f2[keep] / -k2
    v = torch.zeros(f2.shape, dtype=F64, device=DEV)
    beta, step = 1.0, None   # the default relaxation: decay 0.995, TV step 0.2 Dp, reduced by 0.95 past 0.95 Dp

    def consistent(x):
        g = torch.fft.fftn(x.to(C128))
        g[keep] = beta * data + (1 - beta) * g[keep]
        return torch.fft.ifftn(g)

    def tv_gradient(x):
        d = [x - torch.roll(x, 1, ax) for ax in range(3)]
        inv = torch.rsqrt(eps + sum(e * e for e in d))
        g = sum(d) * inv
        for ax in range(3):
            g -= torch.roll(d[ax] * inv, -1, ax)
        return g

    for _ in range(case["iterations"]):
        u = torch.sqrt(1.0 + consistent(v)).real - 1.0
        vp = torch.where(u > 0, u * (2 + u), 0.0)
        dp = float((vp - v).norm())
        step = 0.2 * dp if step is None else step
        v = vp.clone()
        for _ in range(case["tv_steps"]):
            g = tv_gradient(v)
            v = v - step / float(g.norm()) * g
        if float((v - vp).norm()) > 0.95 * dp:
            step *= 0.95
        beta *= 0.995
    return torch.roll(_index(consistent(v), n_med), (f2.shape[0] // 2,) * 3, (0, 1, 2))


def exact(case, seed):
    kind = case["kind"]
    if kind == "tomogram":
        holo, bg, ax, ay = _tomogram_data(case, seed)
        ph, am = _exact_qpi_a(holo, bg, case["n"])
        ph = _exact_unwrap(ph.float(), 0)
        u = _exact_spectra(ph, am, case["n"] // 4, case["n"], case["r"])
        fm0, df, dx, k2 = _geometry(case)
        f2, cnt = _exact_mapping(u, ax, ay, fm0, df, dx)
        return _exact_loop(f2, cnt > 0, case["iterations"], k2, case["accelerated"])
    if kind == "qpi":
        holo, bg, _, _ = _qpi_data(case, seed)
        return (_exact_qpi_a if case["method"] == "a" else _exact_qpi_b)(holo, bg, case["n"])
    if kind == "unwrap":
        return _exact_unwrap(_wrapped(seed, case["maps"], case["m"], case["m"], 12.0, 0.05), case["mode"])
    if kind == "goldstein":
        return None
    if kind == "mapping":
        u = _exact_spectra(*_maps(case, seed), case["m"], case["n"], case["r"])
        fm0, df, dx, _ = _geometry(case)
        return u, _exact_mapping(u, *_angles(case["angles"]), fm0, df, dx)[0], None
    if kind == "loop":
        f2, counts = _kspace(case, seed)
        return _exact_loop(f2.to(C128), counts > 0, case["iterations"], _geometry(case)[3], case["accelerated"])
    if kind == "gradient":
        return _exact_gradient(case, seed)
    f2, _ = _kspace(case, seed, "line")
    return _exact_pocs(f2.to(C128), _geometry(case)[3], case)
