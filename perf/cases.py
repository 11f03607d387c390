"""The work that a user of chromatix_b200 has it do, as measurable cases.

Each case is one call (or one call and its gradient) through the public entry
points of ``chromatix_b200.functional``, ``.systems`` and ``.experimental.mbs``:

  propagate   angular-spectrum / Fresnel-transfer propagation of a stack of fields, padded, with or
              without the gradient of the input field; one or several wavelengths
  rescaled    band-limited propagation onto a grid of another pitch (chirp-Z)
  psf         the widefield PSF stack of a 4f system: point source, phase mask, lens, intensity
  design      the same PSF as a differentiable function of the mask, with the mask's gradient
  multislice  a thick sample slice by slice, with or without the gradient of its refractive index
  microscope  the image of a volume: PSF stack and plane-wise convolution, summed on the sensor
  mbs         iterations of the modified Born series for Maxwell's equations in a box

Everything runs in the default precision ("accurate": FP64 phase arguments, FP32 transforms), the one that
programs use unless they reproduce another package's rounding.
"""

import math

import numpy as np
import torch

DEV = "cuda"
TAU = 2 * math.pi


# ---------------------------------------------------------------------------------------------------------
# the cases
# ---------------------------------------------------------------------------------------------------------
def listed():
    return [
        # one small field, as an interactive program or an alignment loop propagates it: latency
        dict(name="asm_256_one", kind="propagate", method="asm", batch=1, ny=256, nx=256, pad_y=128, pad_x=128,
             wv=1, mode="same", bandlimit=False, grad=False),
        # a stack of independent fields, twofold padding: holograms of a sequence, modes of a source
        dict(name="asm_512_x64", kind="propagate", method="asm", batch=64, ny=512, nx=512, pad_y=256, pad_x=256,
             wv=1, mode="full", bandlimit=False, grad=False),
        # colour holograms on a display's grid: not square, the three wavelengths innermost
        dict(name="transfer_rgb_600x800", kind="propagate", method="transfer", batch=4, ny=600, nx=800, pad_y=84,
             pad_x=112, wv=3, mode="same", bandlimit=False, grad=False),
        # a camera's crop of odd size with the padding that the distance asks for: no smooth transform length
        dict(name="asm_odd_501x675", kind="propagate", method="asm", batch=2, ny=501, nx=675, pad_y=100, pad_x=120,
             wv=1, mode="same", bandlimit=False, grad=False),
        # phase retrieval: a propagation and its gradient, for a few recordings at once
        dict(name="asm_grad_640_x8", kind="propagate", method="asm", batch=8, ny=640, nx=640, pad_y=192, pad_x=192,
             wv=1, mode="same", bandlimit=False, grad=True),
        # one field at the highest resolution, band-limited: the reference's own large example
        dict(name="asm_4096_bandlimit", kind="propagate", method="asm", batch=1, ny=4096, nx=4096, pad_y=2048,
             pad_x=2048, wv=1, mode="same", bandlimit=True, grad=False),
        # a zoom onto a detector of finer pitch: the reference's rescaled example
        dict(name="rescaled_1024", kind="rescaled", ny=1024, nx=1024, pad=512, my=1024, mx=1024, zoom=4.0),
        # the headline: a colour PSF stack of a widefield microscope
        dict(name="psf_1280_z64_rgb", kind="psf", n=1280, nz=64, wv=3, NA=0.6),
        # PSF engineering: the gradient of a PSF stack with respect to its phase mask
        dict(name="design_768_z16", kind="design", n=768, nz=16, wv=1, NA=0.8),
        # tomography: a thick sample's field and the gradient of its refractive index
        dict(name="multislice_grad_1024x128", kind="multislice", n=1024, pad=0, slices=128, grad=True),
        # the reference's imaging benchmark: a volume through its PSF stack onto a camera
        dict(name="microscope_1536x128", kind="microscope", n=1536, nz=128),
        # full-vector scattering in a box with absorbing walls, a few iterations of the series
        dict(name="mbs_320", kind="mbs", X=320, Y=320, Z=320, iterations=10),
    ]


def _sizes(lo, hi):
    """Even transform lengths 2^a {1, 3, 5, 7} in [lo, hi]: what PSF, slice and box grids are made of."""
    return sorted(q * 2**a for q in (1, 3, 5, 7) for a in range(1, 14) if lo <= q * 2**a <= hi)


def _log_int(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    kind = rng.choice(["propagate", "propagate", "propagate", "rescaled", "psf", "design", "multislice",
                       "multislice", "microscope", "mbs"])
    if kind == "propagate":
        ny, nx = _log_int(rng, 150, 1500), _log_int(rng, 150, 1500)
        if rng.random() < 0.7:  # padded to a smooth grid, as most programs do
            ny, nx = ny + ny % 2, nx + nx % 2
            py = rng.choice([s for s in _sizes(ny, 2 * ny + 16) if s >= 1.2 * ny])
            px = rng.choice([s for s in _sizes(nx, 2 * nx + 16) if s >= 1.2 * nx])
            pad_y, pad_x = (py - ny) // 2, (px - nx) // 2
        else:  # padded by whatever the distance asks for
            pad_y, pad_x = rng.randint(ny // 10, ny // 2), rng.randint(nx // 10, nx // 2)
        wv = rng.choice([1, 1, 1, 2, 3])
        room = 64 * 1024 * 1024 // ((ny + 2 * pad_y) * (nx + 2 * pad_x) * wv)
        return dict(kind=kind, method=rng.choice(["asm", "transfer"]), batch=_log_int(rng, 1, max(1, min(64, room))),
                    ny=ny, nx=nx, pad_y=pad_y, pad_x=pad_x, wv=wv, mode=rng.choice(["same", "full"]),
                    bandlimit=False, grad=rng.random() < 0.4)
    if kind == "rescaled":
        n = rng.choice(_sizes(256, 1280))
        pad = n // 2 if rng.random() < 0.7 else 0
        return dict(kind=kind, ny=n, nx=n, pad=pad, my=_log_int(rng, 200, 1400), mx=_log_int(rng, 200, 1400),
                    zoom=round(rng.uniform(1.5, 8.0), 2))
    if kind in ("psf", "design"):
        n = rng.choice(_sizes(256, 1536 if kind == "psf" else 1024))
        wv = rng.choice([1, 3])
        most = (64 * 3 * 1280 * 1280 if kind == "psf" else 40 * 768 * 768) // (n * n * wv)
        return dict(kind=kind, n=n, nz=_log_int(rng, 2, max(3, min(128, most))), wv=wv,
                    NA=round(rng.uniform(0.3, 0.9), 2))
    if kind == "multislice":
        n = rng.choice(_sizes(256, 1024))
        grad = rng.random() < 0.5
        pad = rng.choice([0, n // 8 if (n + n // 4) in _sizes(256, 1280) else 0])
        most = 128 * 1024 * 1024 // ((n + 2 * pad) ** 2)
        return dict(kind=kind, n=n, pad=pad, slices=_log_int(rng, 8, max(9, min(200, most))), grad=grad)
    if kind == "microscope":
        n = rng.choice(_sizes(256, 1536))
        return dict(kind=kind, n=n, nz=_log_int(rng, 4, max(5, min(128, 128 * 1536 * 1536 // (n * n)))))
    X, Y, Z = (rng.choice(_sizes(96, 320)) for _ in range(3))
    return dict(kind="mbs", X=X, Y=Y, Z=Z, iterations=rng.randint(4, 10))


# ---------------------------------------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------------------------------------
def _gen(seed):
    g = torch.Generator(device=DEV)
    g.manual_seed(int(seed))
    return g


def _rand(g, *shape):
    return torch.rand(shape, generator=g, device=DEV, dtype=torch.float32)


def _fields(g, *shape):
    """Complex fields of amplitude in [0.5, 1) and any phase."""
    return torch.polar(0.5 + 0.5 * _rand(g, *shape), TAU * _rand(g, *shape))


def _wavelengths(wv):
    return [0.532] if wv == 1 else [float(v) for v in np.linspace(0.45, 0.63, wv)]


def _smooth(g, depth, n, sigma):
    """(depth, n, n) of unit-variance noise, periodic Gaussian filter of `sigma` pixels slice by slice."""
    f = torch.fft.fftfreq(n, device=DEV)
    k = torch.exp(-0.5 * (TAU * sigma) ** 2 * (f[:, None] ** 2 + f[None, :] ** 2))
    out = torch.empty((depth, n, n), device=DEV)
    for i in range(depth):
        out[i] = torch.fft.ifft2(torch.fft.fft2(torch.randn((n, n), generator=g, device=DEV)) * k).real
    return out


PROP = dict(z=100.0, n=1.33, dx=0.3)
LENS = dict(f_obj=8000.0, f_tube=200000.0, n=1.33, pitch=6.5)
SLICE = dict(dz=0.2, dx=0.1, lam=0.532, n=1.33, NA=0.8)
BOX = dict(spacing=0.1, lam=0.5, n=1.33, wall=16)
SCOPE = dict(spacing=0.3, f=100.0, n=1.33, NA=0.8, lam=0.532)
DETECTOR = dict(lam=0.532, dx=1.064, n=1.0)


def _psf_dx(case):
    """Pupil spacing per wavelength that gives the camera's pitch after the tube lens."""
    wl = np.asarray(_wavelengths(case["wv"]))
    return LENS["f_tube"] * wl / (LENS["n"] * case["n"] * LENS["pitch"])


def _psf_planes(g, nz):
    return torch.sort(10.0 * _rand(g, nz).double() - 5.0).values


def _rescaled_geometry(case):
    D = DETECTOR["dx"] * case["ny"]
    return 10 * D, DETECTOR["dx"] / case["zoom"], (0.0, D / 20)


def _mbs_index(g, case):
    """Refractive index of the inner box: spheres in a medium."""
    w = BOX["wall"]
    shape = [case[k] - 2 * w for k in "XYZ"]
    ax = [(torch.arange(s, device=DEV, dtype=torch.float32) - s // 2) * BOX["spacing"] for s in shape]
    r = torch.rand((60, 5), generator=g, device=DEV).cpu().tolist()
    n = torch.full(shape, BOX["n"], device=DEV)
    for a, b, c, d, e in r:
        ctr = [(v - 0.5) * s * BOX["spacing"] for v, s in zip((a, b, c), shape)]
        d2 = (ax[0][:, None, None] - ctr[0]) ** 2 + (ax[1][None, :, None] - ctr[1]) ** 2 + (ax[2][None, None, :] - ctr[2]) ** 2
        n = torch.where(d2 <= (0.4 + 1.6 * d) ** 2, torch.full_like(n, 1.36 + 0.09 * e), n)
    return n


def prepare(case, seed):
    from chromatix_b200.core.field import ChromaticScalarField, ScalarField
    from chromatix_b200.core.spectrum import Spectrum

    g, kind = _gen(seed), case["kind"]
    s = {"case": case}
    if kind in ("propagate", "rescaled"):
        B, W = case.get("batch", 1), case.get("wv", 1)
        shape = ((B,) if B > 1 else ()) + (case["ny"], case["nx"]) + ((W,) if W > 1 else ())
        u = _fields(g, *shape)
        if kind == "rescaled":
            s["field"] = ScalarField(u, DETECTOR["dx"], 0.0, Spectrum.build(DETECTOR["lam"]))
            return s
        if case["grad"]:
            u.requires_grad_(True)
            py, px = 2 * case["pad_y"], 2 * case["pad_x"]
            if case["mode"] == "same":
                py = px = 0
            d = 1 if B > 1 else 0
            s["cotangent"] = _fields(g, *shape[:d], shape[d] + py, shape[d + 1] + px, *shape[d + 2:])
        if W > 1:
            s["field"] = ChromaticScalarField(u, PROP["dx"], 0.0, Spectrum.build(np.asarray(_wavelengths(W))))
        else:
            s["field"] = ScalarField(u, PROP["dx"], 0.0, Spectrum.build(_wavelengths(1)[0]))
    elif kind in ("psf", "design"):
        s["z"] = _psf_planes(g, case["nz"])
        s["phase"] = TAU * _rand(g, case["n"], case["n"])
        if kind == "design":
            s["phase"].requires_grad_(True)
            s["cotangent"] = _rand(g, case["nz"], case["n"], case["n"])
    elif kind == "multislice":
        n, D = case["n"], case["slices"]
        s["dn"] = 0.3 * _smooth(g, D, n, 4.0)
        s["ab"] = _rand(g, D, n, n) * (0.05 / (TAU / SLICE["lam"] * SLICE["dz"]))
        u = torch.polar(torch.ones((n, n), device=DEV), 0.5 * _smooth(g, 1, n, 8.0)[0])
        s["field"] = ScalarField(u, SLICE["dx"], 0.0, Spectrum.build(SLICE["lam"]))
        if case["grad"]:
            s["dn"].requires_grad_(True)
            s["cotangent"] = _fields(g, n, n)
    elif kind == "microscope":
        from chromatix_b200.systems import BasicSensor, Microscope, Optical4FSystemPSF

        n = case["n"]
        s["volume"] = _rand(g, case["nz"], n, n)
        s["z"] = _psf_planes(g, case["nz"]) * 0.8
        s["phase"] = TAU * _rand(g, n, n)
        s["scope"] = Microscope(Optical4FSystemPSF((n, n), SCOPE["spacing"], SCOPE["f"], s["phase"]),
                                BasicSensor((n, n), SCOPE["spacing"], resampling_method=None, reduce_axis=0),
                                SCOPE["f"], SCOPE["n"], SCOPE["NA"], SCOPE["lam"])
    else:
        from chromatix_b200.experimental import mbs

        eps = (_mbs_index(g, case) ** 2).to(torch.complex64)
        s["sample"] = mbs.add_absorbing_bc(mbs.Sample(eps, BOX["spacing"]), (0, 1, 2), (BOX["wall"] + 0.5) * BOX["spacing"],
                                           0.25, BOX["n"])
        J = torch.zeros(tuple(s["sample"].shape) + (3,), dtype=torch.complex64, device=DEV)
        J[BOX["wall"] + 2, :, :, 1] = 1.0
        s["source"] = mbs.Source(J, TAU / BOX["lam"])
        s["shift"], s["scale"] = mbs.get_shift_and_scale(s["sample"].permittivity)
    return s


# ---------------------------------------------------------------------------------------------------------
# one pass
# ---------------------------------------------------------------------------------------------------------
def run(s):
    import chromatix_b200.functional as cf

    case = s["case"]
    kind = case["kind"]
    if kind == "propagate":
        f = s["field"]
        pad = (case["pad_y"], case["pad_x"])
        if case["method"] == "asm":
            out = cf.asm_propagate(f, PROP["z"], PROP["n"], pad, bandlimit=case["bandlimit"], mode=case["mode"])
        else:
            out = cf.transfer_propagate(f, PROP["z"], PROP["n"], pad, mode=case["mode"])
        if not case["grad"]:
            return out.u
        (gu,) = torch.autograd.grad(out.u, f.u, s["cotangent"])
        return [out.u.detach(), gu]
    if kind == "rescaled":
        z, dx, shift = _rescaled_geometry(case)
        pad = (case["pad"], case["pad"])
        return cf.asm_propagate(s["field"], z, DETECTOR["n"], pad, bandlimit=True, output_dx=np.full_like(s["field"].dx, dx),
                                output_shape=(case["my"], case["mx"]), shift_yx=shift, mode="full").u
    if kind in ("psf", "design"):
        wl = _wavelengths(case["wv"])
        dx = _psf_dx(case)
        spec = (np.asarray(wl), np.ones(len(wl))) if len(wl) > 1 else wl[0]
        n = case["n"]
        f = cf.objective_point_source((n, n), dx if len(wl) > 1 else float(dx[0]), spec, s["z"], LENS["f_obj"],
                                      LENS["n"], case["NA"], device=DEV)
        I = cf.ff_lens(cf.phase_change(f, s["phase"]), LENS["f_tube"], LENS["n"]).intensity
        if kind == "psf":
            return I
        (gp,) = torch.autograd.grad(I, s["phase"], s["cotangent"])
        return [I.detach(), gp]
    if kind == "multislice":
        out = cf.multislice_thick_sample(s["field"], s["ab"], s["dn"], SLICE["n"], SLICE["dz"], case["pad"],
                                         NA=SLICE["NA"])
        if not case["grad"]:
            return out.u
        (gn,) = torch.autograd.grad(out.u, s["dn"], s["cotangent"])
        return [out.u.detach(), gn]
    if kind == "microscope":
        return s["scope"](s["volume"], s["z"])
    from chromatix_b200.experimental import mbs

    return mbs.solve(s["sample"], s["source"], maxiter=case["iterations"], tol=0.0, shift=s["shift"], scale=s["scale"])


# ---------------------------------------------------------------------------------------------------------
# what a pass cannot do without
# ---------------------------------------------------------------------------------------------------------
def _fft(n):
    return 5.0 * n * math.log2(max(n, 2))


def work(case):
    kind = case["kind"]
    if kind == "propagate":
        B = case["batch"] * case["wv"]
        P = (case["ny"] + 2 * case["pad_y"]) * (case["nx"] + 2 * case["pad_x"])
        n = case["ny"] * case["nx"]
        out = n if case["mode"] == "same" else P
        k = 2 if case["grad"] else 1
        return {"bytes": 8.0 * B * (n + out) * k, "flops": k * B * (2 * _fft(P) + 6 * P)}
    if kind == "rescaled":
        Py, Px = case["ny"] + 2 * case["pad"], case["nx"] + 2 * case["pad"]
        my, mx = case["my"], case["mx"]
        ly, lx = Py + my, Px + mx
        return {"bytes": 8.0 * (case["ny"] * case["nx"] + my * mx),
                "flops": _fft(Py * Px) + 2 * Px * _fft(ly) + 2 * my * _fft(lx)}
    if kind in ("psf", "design"):
        n2, nz, W = case["n"] ** 2, case["nz"], case["wv"]
        k = 2 if kind == "design" else 1
        return {"bytes": 4.0 * (n2 * k + nz * n2 * k), "flops": k * nz * W * (_fft(n2) + 10 * n2)}
    if kind == "multislice":
        n2, D = case["n"] ** 2, case["slices"]
        P = (case["n"] + 2 * case["pad"]) ** 2
        k = 2 if case["grad"] else 1
        maps = 3 if case["grad"] else 2
        return {"bytes": 4.0 * maps * D * n2 + 16.0 * n2 * k, "flops": k * D * (2 * _fft(P) + 20 * P)}
    if kind == "microscope":
        n, nz = case["n"], case["nz"]
        return {"bytes": 4.0 * (nz * n * n + 2 * n * n),
                "flops": nz * (_fft(n * n) + 10 * n * n + _fft(4 * n * n) + 8 * n * n)}
    v = case["X"] * case["Y"] * case["Z"]
    return {"bytes": 8.0 * v * (1 + 3 + 3), "flops": case["iterations"] * v * (6 * 5.0 * math.log2(v) + 120)}


# ---------------------------------------------------------------------------------------------------------
# the same values in 64 bits, from the formulas
# ---------------------------------------------------------------------------------------------------------
def _freq(n, dx):
    return torch.fft.fftfreq(n, dx, dtype=torch.float64, device=DEV)


def _asm(py, px, dy, dx, z, lam, n, bandlimit=False):
    """Angular-spectrum transfer function on the FFT grid; waves past the cutoff decay."""
    fy, fx = _freq(py, dy)[:, None], _freq(px, dx)[None, :]
    k = (1 - (lam / n) ** 2 * (fy**2 + fx**2)).to(torch.complex128)
    h = torch.exp(1j * (TAU * abs(z) * n / lam) * torch.sqrt(k))
    h = h if z >= 0 else h.conj()
    if bandlimit:  # the highest frequency that the sampling of the transfer function allows, per axis
        for f, m, d in ((fy, py, dy), (fx, px, dx)):
            h = h * (f.abs() <= 1 / (lam * math.sqrt((2 * abs(z) / (m * d)) ** 2 + 1)))
    return h


def _fresnel(py, px, dy, dx, z, lam, n):
    fy, fx = _freq(py, dy)[:, None], _freq(px, dx)[None, :]
    return torch.exp(-1j * (math.pi * lam * z / n) * (fy**2 + fx**2).to(torch.complex128))


def _exact_propagate(case, s):
    B, W = case["batch"], case["wv"]
    ny, nx, cy, cx = case["ny"], case["nx"], case["pad_y"], case["pad_x"]
    py, px = ny + 2 * cy, nx + 2 * cx
    same = case["mode"] == "same"

    def through(u, adjoint):
        u = u.detach().reshape((B,) + tuple(u.shape[(1 if B > 1 else 0):][:2]) + (W,))
        pad_in, pad_out = (True, same) if not adjoint else (same, True)
        oy, ox = (ny, nx) if pad_out else (py, px)
        out = torch.empty((B, oy, ox, W), dtype=torch.complex128, device=DEV)
        for w, lam in enumerate(_wavelengths(W)):
            if case["method"] == "asm":
                h = _asm(py, px, PROP["dx"], PROP["dx"], PROP["z"], lam, PROP["n"], case["bandlimit"])
            else:
                h = _fresnel(py, px, PROP["dx"], PROP["dx"], PROP["z"], lam, PROP["n"])
            h = h.conj() if adjoint else h
            for b in range(B):
                v = u[b, :, :, w].to(torch.complex128)
                if pad_in:
                    v = torch.nn.functional.pad(v, (cx, cx, cy, cy))
                v = torch.fft.ifft2(torch.fft.fft2(v) * h)
                out[b, :, :, w] = v[cy:cy + ny, cx:cx + nx] if pad_out else v
        out = out if W > 1 else out[..., 0]
        return out if B > 1 else out[0]

    out = through(s["field"].u, False)
    return [out, through(s["cotangent"], True)] if case["grad"] else out


def _exact_rescaled(case, s):
    lam, dx, n = DETECTOR["lam"], DETECTOR["dx"], DETECTOR["n"]
    z, dxo, shift = _rescaled_geometry(case)
    p = case["pad"]
    u = torch.nn.functional.pad(s["field"].u.to(torch.complex128), (p, p, p, p))
    py, px = u.shape
    sp = torch.fft.fftshift(_asm(py, px, dx, dx, z, lam, n, True) * torch.fft.fft2(torch.fft.ifftshift(u)))
    kern = []
    for m, P, sh in ((case["my"], py, shift[0]), (case["mx"], px, shift[1])):
        T = P * dx
        x = dxo * (torch.arange(m, dtype=torch.float64, device=DEV) - m / 2) + sh
        j = torch.arange(P, dtype=torch.float64, device=DEV) - (m - 1) // 2
        ph = torch.remainder(x[:, None] * j[None, :] / T, 1.0)
        kern.append(torch.polar(torch.full_like(ph, 1 / (dxo * T)), TAU * ph))
    return kern[0] @ sp @ kern[1].T


def _exact_pupil(n, dx, radius):
    r = dx * (torch.arange(n, dtype=torch.float64, device=DEV) - n / 2)
    r2 = r[:, None] ** 2 + r[None, :] ** 2
    return r2, r2 <= radius**2


def _exact_psf(n, wls, dxs, zs, phase, f_obj, f_tube, med, NA):
    """Intensity of every plane, as a list; phase may need a gradient."""
    dens = 1.0 / len(wls)
    parts, pw = [], 0.0
    for lam, dx in zip(wls, dxs):
        L2 = lam * f_obj / med
        r2, inside = _exact_pupil(n, dx, wls[0] / lam * f_obj * NA / med)
        parts.append((lam, dx, L2, r2, inside))
        pw += dens * float(inside.sum()) / L2**2
    out = []
    for z in zs.tolist():
        I = 0.0
        for lam, dx, L2, r2, inside in parts:
            amp = 1 / L2 / math.sqrt(pw * dx * dx) * (dx * dx) / (lam * f_tube / med)
            ph = (-math.pi * (z / f_obj) / L2) * r2 + phase * (wls[0] / lam)
            u = torch.polar(inside.double() * amp, ph)
            I = I + dens * torch.fft.fftshift(torch.fft.fft2(torch.fft.ifftshift(u)).abs().square())
        out.append(I)
    return out


def _exact_multislice(case, s):
    n, p, D = case["n"], case["pad"], case["slices"]
    lam, dz, dx, med = SLICE["lam"], SLICE["dz"], SLICE["dx"], SLICE["n"]
    P = n + 2 * p
    k = TAU / lam
    H = _asm(P, P, dx, dx, dz, lam, med)
    Hd = _asm(P, P, dx, dx, -dz * D / 2, lam, med)
    f2 = _freq(P, dx)[:, None] ** 2 + _freq(P, dx)[None, :] ** 2
    Hd = Hd * (f2 <= (SLICE["NA"] / lam) ** 2)
    pad = lambda v: torch.nn.functional.pad(v, (p, p, p, p))  # noqa: E731
    dn, ab = s["dn"].detach(), s["ab"]

    def t(i):
        a = pad(ab[i].double())
        return torch.polar(torch.exp(-k * dz * a), k * dz * pad(dn[i].double()))

    u = pad(s["field"].u.to(torch.complex128))
    kept = []
    for i in range(D):
        u = torch.fft.ifft2(torch.fft.fft2(u) * H) * t(i)
        if case["grad"]:
            kept.append(u)
    out = torch.fft.ifft2(torch.fft.fft2(u) * Hd)[p:p + n, p:p + n]
    if not case["grad"]:
        return out
    g = torch.fft.ifft2(torch.fft.fft2(pad(s["cotangent"].to(torch.complex128))) * Hd.conj())
    gn = torch.empty((D, n, n), dtype=torch.float64, device=DEV)
    for i in reversed(range(D)):
        gn[i] = (k * dz * (g * kept[i].conj()).imag)[p:p + n, p:p + n]
        g = torch.fft.ifft2(torch.fft.fft2(g * t(i).conj()) * H.conj())
    return [out, gn]


def _exact_microscope(case, s):
    n = case["n"]
    dx = SCOPE["f"] * SCOPE["lam"] / (SCOPE["n"] * n * SCOPE["spacing"])
    acc = 0.0
    phase = s["phase"].double()
    for i in range(case["nz"]):
        (psf,) = _exact_psf(n, [SCOPE["lam"]], [dx], s["z"][i:i + 1], phase, SCOPE["f"], SCOPE["f"], SCOPE["n"], SCOPE["NA"])
        acc = acc + torch.fft.rfft2(s["volume"][i].double(), (2 * n, 2 * n)) * torch.fft.rfft2(psf, (2 * n, 2 * n))
    o = (n - 1) // 2
    return torch.fft.irfft2(acc, (2 * n, 2 * n))[o:o + n, o:o + n].contiguous()


def _exact_mbs(case, s):
    k0 = TAU / BOX["lam"]
    eps = s["sample"].permittivity.to(torch.complex128)
    src = s["source"].field.to(torch.complex128).movedim(-1, 0)
    c, bias = complex(s["scale"]), complex(s["shift"])
    kb = bias * c + 1
    k = [TAU * _freq(m, BOX["spacing"]) / k0 for m in eps.shape]
    k = [k[0][:, None, None], k[1][None, :, None], k[2][None, None, :]]
    k2 = k[0] ** 2 + k[1] ** 2 + k[2] ** 2
    V = c * eps - kb
    inv = 1 / (kb - c * k2)
    k2i = torch.where(k2 > 0, 1 / torch.where(k2 > 0, k2, 1.0), 0.0)

    def green(y):
        y = torch.fft.fftn(y, dim=(1, 2, 3))
        pr = (k[0] * y[0] + k[1] * y[1] + k[2] * y[2]) * k2i
        y = torch.stack([(y[a] - k[a] * pr) * inv + k[a] * pr / kb for a in range(3)])
        return torch.fft.ifftn(y, dim=(1, 2, 3))

    b = -V * green(src * c)
    top = float(b.abs().max())
    b = b / top
    x = b
    for _ in range(case["iterations"]):
        x = b + V * (green(V * x) + x) + x
    return (x * top).movedim(0, -1).contiguous()


def exact(case, seed):
    s = prepare(case, seed)
    kind = case["kind"]
    if kind == "propagate":
        return _exact_propagate(case, s)
    if kind == "rescaled":
        return _exact_rescaled(case, s)
    if kind == "psf":
        return torch.stack(_exact_psf(case["n"], _wavelengths(case["wv"]), _psf_dx(case).tolist(), s["z"], s["phase"].double(),
                                      LENS["f_obj"], LENS["f_tube"], LENS["n"], case["NA"]))
    if kind == "design":
        ph = s["phase"].detach().double().requires_grad_(True)
        g = torch.zeros_like(ph)
        planes = []
        for i in range(case["nz"]):
            (I,) = _exact_psf(case["n"], _wavelengths(case["wv"]), _psf_dx(case).tolist(), s["z"][i:i + 1], ph, LENS["f_obj"],
                              LENS["f_tube"], LENS["n"], case["NA"])
            g = g + torch.autograd.grad(I, ph, s["cotangent"][i].double())[0]
            planes.append(I.detach())
        return [torch.stack(planes), g]
    if kind == "multislice":
        return _exact_multislice(case, s)
    if kind == "microscope":
        return _exact_microscope(case, s)
    return _exact_mbs(case, s)
