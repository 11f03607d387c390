"""GPU: the propagation passes on pairs of rows and columns, at every length
with a plan, rows of odd length, odd numbers of rows, and each way the
propagator is applied.

Tolerance: an FP32 transform of length N rounds with a relative L2 error of
about 0.5 eps sqrt(log2 N) <= 1.1e-7, four of them 2.2e-7 added in squares; the
propagator's hardware sin / cos adds at most 4e-7 (absolute, |H| <= 1).  The
bar is twice their sum, 1.3e-6.
"""

import numpy as np
import pytest

from oracle import chromatix_oracle as O

pytestmark = pytest.mark.gpu

BAR = 1.3e-6
LENGTHS = [128, 160, 192, 224, 256, 320, 384, 448, 512, 640, 768, 896, 1024, 1280, 1536, 1792, 2048, 2560, 3072, 3584,
           4096, 8192]


def to_cuda(a):
    import torch

    return torch.as_tensor(a, device="cuda")


def _field(u, dx=0.3, lam=0.532):
    from chromatix_b200.core.field import ChromaticScalarField, ScalarField
    from chromatix_b200.core.spectrum import Spectrum

    spec = Spectrum.build(lam)
    cls = ChromaticScalarField if spec.size > 1 else ScalarField
    return cls(to_cuda(u), dx, 0.0, spec)


def _crand(rng, shape):
    return (rng.standard_normal(shape) + 1j * rng.standard_normal(shape)).astype(np.complex64)


@pytest.mark.parametrize("n", LENGTHS)
def test_table_propagator_every_length(n):
    import chromatix_b200.functional as cf

    rng = np.random.default_rng(n)
    # columns of length n with a ragged last tile (10 columns), with odd rows (5), and rows of length n
    for shape in ((n, 10), (n, 5), (6, n)):
        u = _crand(rng, (3,) + shape)
        H = _crand(rng, shape)
        out = cf.kernel_propagate(_field(u), to_cuda(H)).u.cpu().numpy()
        ref = np.fft.ifft2(np.fft.fft2(u.astype(np.complex128)) * H)
        assert O.rel_l2(out, ref) < BAR, shape


@pytest.mark.parametrize("n", LENGTHS)
def test_evaluated_propagator_every_length(n):
    import chromatix_b200.functional as cf

    rng = np.random.default_rng(n + 1)
    z = [40.0, 40.0, -15.0]  # a plane with its predecessor's propagator, then another
    # padded on both sides, an odd number of data rows never divides into pairs
    for ny, nx, pad in ((n - 2 * (n // 5), 4, (n // 5, 1)), (n // 2, 6, (n // 4, 0))):
        u = _crand(rng, (3, ny, nx))
        f = _field(u)
        for kw in (dict(mode="same"), dict(mode="full", shift_yx=(1.5, -0.7)), dict(mode="full", kykx=(0.2, 0.1))):
            out = cf.asm_propagate(f, np.array(z), 1.33, pad, **kw).u.cpu().numpy()
            for b in range(3):
                ref = O.asm_propagate(O.field_build(u[b], 0.3, 0.532), z[b], 1.33, pad, **kw).u
                assert O.rel_l2(out[b], np.asarray(ref).reshape(out[b].shape)) < BAR, (ny, kw, b)


@pytest.mark.parametrize("ny,nx,pad", [(101, 131, (21, 29)), (77, 96, (26, 16))])
def test_odd_rows_and_wavelengths(ny, nx, pad):
    """Odd numbers of rows with two wavelengths innermost, forward and gradient."""
    import torch

    import chromatix_b200.functional as cf

    # padded to lengths with a plan (odd fields: odd padded lengths go another way, so pad unevenly sized fields)
    ny, nx = ny + ny % 2, nx + nx % 2
    rng = np.random.default_rng(5)
    u = _crand(rng, (2, ny, nx, 2))
    lam = np.array([0.45, 0.6])
    f = _field(u, lam=lam)
    f.u.requires_grad_(True)
    py = min(n for n in LENGTHS if n >= ny + pad[0])
    px = min(n for n in LENGTHS if n >= nx + pad[1])
    pads = ((py - ny) // 2, (px - nx) // 2)
    out = cf.transfer_propagate(f, 30.0, 1.33, pads, mode="same")
    g = _crand(rng, out.u.shape)
    (gu,) = torch.autograd.grad(out.u, f.u, to_cuda(g))
    for w in range(2):
        fy, fx = np.fft.fftfreq(py, 0.3), np.fft.fftfreq(px, 0.3)
        H = np.exp(-1j * np.pi * lam[w] * 30.0 / 1.33 * (fy[:, None] ** 2 + fx[None, :] ** 2))
        for src, h, dst in ((u, H, out.u.detach().cpu().numpy()), (g, H.conj(), gu.cpu().numpy())):
            for b in range(2):
                v = np.pad(src[b, :, :, w].astype(np.complex128), [(p, p) for p in pads])
                ref = np.fft.ifft2(np.fft.fft2(v) * h)[pads[0]:pads[0] + ny, pads[1]:pads[1] + nx]
                assert O.rel_l2(dst[b, :, :, w], ref) < BAR


@pytest.mark.parametrize("ny,nx,wv", [(128, 128, 3), (160, 10, 1), (224, 5, 2), (320, 448, 1), (768, 256, 2),
                                      (1280, 192, 3), (2048, 128, 1), (192, 4096, 1), (4096, 128, 2)])
def test_psf_stack(ny, nx, wv):
    """The fused PSF: stored row spectra of odd and even pitch, row boxes of odd height, an offset source, one and
    several wavelengths (tolerance of the intensity: twice the field's, and the source's sin / cos are FP64)."""
    import chromatix_b200.functional as cf

    rng = np.random.default_rng(ny + nx)
    wl = np.array([0.532, 0.45, 0.63][:wv])
    dx = 8000.0 * 0.532 / (1.33 * 0.35 * min(ny, nx)) * 0.01 * (wl / 0.532)
    z = np.array([-3.0, 0.5, 4.0])
    spec = (wl, np.arange(1.0, wv + 1)) if wv > 1 else float(wl[0])
    phase = rng.uniform(0, 2 * np.pi, (ny, nx)).astype(np.float32)
    NA = 0.8 * 1.33 * min(ny, nx) / 2 * float(dx.min()) / 8000.0  # a pupil of 0.8 of the shorter side
    args = ((ny, nx), dx if wv > 1 else float(dx[0]), spec, z, 8000.0, 1.33, NA)
    off = (0.3 * float(dx[0]), -0.2 * float(dx[0]))
    f = cf.objective_point_source(*args, offset=off, device="cuda")
    out = cf.ff_lens(cf.phase_change(f, to_cuda(phase)), 200000.0, 1.33).intensity.cpu().numpy()
    ref = O.ff_lens(O.phase_change(O.objective_point_source(*args, offset=off), phase), 200000.0, 1.33).intensity
    assert O.rel_l2(out, np.asarray(ref).reshape(out.shape)) < 2 * BAR


@pytest.mark.parametrize("planes,h,w,kh,kw", [(3, 64, 128, 64, 128), (2, 101, 190, 101, 190), (4, 75, 333, 60, 330),
                                              (2, 300, 131, 305, 140), (1, 700, 129, 700, 129), (2, 130, 2048, 131, 2047),
                                              (2, 2048, 130, 2048, 130)])
def test_convolution_pairs(planes, h, w, kh, kw):
    """Sample and kernel as a pair: odd numbers of rows (a row of zeros completes the last pair), odd widths (element
    by element loads), unequal shapes, the longest lengths; per plane and summed.  Four FP32 transforms of each input
    and products: the propagation's tolerance without the sin / cos, doubled for the sum over planes."""
    from chromatix_b200.ops import fourier_convolution

    rng = np.random.default_rng(h + w)
    a = rng.standard_normal((planes, h, w)).astype(np.float32)
    k = rng.standard_normal((planes, kh, kw)).astype(np.float32)
    P, Q = h + kh, w + kw
    F = np.fft.rfft2(a.astype(np.float64), (P, Q)) * np.fft.rfft2(k.astype(np.float64), (P, Q))
    y0, x0 = (kh - 1) // 2, (kw - 1) // 2
    ref = np.fft.irfft2(F, (P, Q))[:, y0:y0 + h, x0:x0 + w]
    out = fourier_convolution(to_cuda(a), to_cuda(k)).cpu().numpy()
    assert O.rel_l2(out, ref) < BAR
    red = fourier_convolution(to_cuda(a), to_cuda(k), reduce=True).cpu().numpy()
    assert O.rel_l2(red, ref.sum(0)) < BAR
    # one kernel for every plane
    one = fourier_convolution(to_cuda(a), to_cuda(k[:1])).cpu().numpy()
    F1 = np.fft.rfft2(a.astype(np.float64), (P, Q)) * np.fft.rfft2(k[:1].astype(np.float64), (P, Q))
    assert O.rel_l2(one, np.fft.irfft2(F1, (P, Q))[:, y0:y0 + h, x0:x0 + w]) < BAR


@pytest.mark.parametrize("ny,nx,pad,wv", [(128, 160, (0, 0), 1), (192, 6, (0, 0), 2), (224, 5, (0, 0), 1), (256, 320, (64, 32), 3),
                                          (320, 10, (32, 1), 1), (2048, 10, (0, 0), 2)])
def test_optical_fft_passes(ny, nx, pad, wv):
    """The chirped optical FFT on pairs: plain (ff_lens with a pupil, inverse lens), with an output chirp (df_lens),
    with chirps, padding and crop (transform_propagate); two transforms and FP64-reduced chirps."""
    import chromatix_b200.functional as cf

    rng = np.random.default_rng(ny + nx)
    lam = np.array([0.532, 0.45, 0.63][:wv])
    spec = lam if wv > 1 else float(lam[0])
    u = _crand(rng, (2, ny, nx) + ((wv,) if wv > 1 else ()))
    f = _field(u, dx=1.1, lam=spec)
    calls = [lambda m, g: m.ff_lens(g, 500.0, 1.33, NA=0.05), lambda m, g: m.ff_lens(g, 500.0, 1.33, inverse=True),
             lambda m, g: m.df_lens(g, 420.0, 500.0, 1.33), lambda m, g: m.transform_propagate(g, 3000.0, 1.0, pad)]
    for i, call in enumerate(calls):
        out = call(cf, f).u.cpu().numpy()
        for b in range(2):
            ref = call(O, O.field_build(u[b], 1.1, spec)).u
            assert O.rel_l2(out[b], np.asarray(ref).reshape(out[b].shape)) < BAR, (i, b)


@pytest.mark.parametrize("n,pad,slices", [(128, 0, 5), (130, 15, 4), (100, 14, 3), (224, 0, 3), (320, 32, 3), (448, 0, 2),
                                          (1024, 0, 2), (1280, 0, 2), (2048, 0, 1)])
def test_multislice_rows(n, pad, slices):
    """The slice loop's row passes on pairs: sides that 4 does not divide (rows read element by element), padding,
    with and without recomputation.  Each slice adds two transforms each way; gradients within twice the field's bar."""
    import torch

    import chromatix_b200.functional as cf

    if n + 2 * pad not in LENGTHS:
        pad = (min(m for m in LENGTHS if m > n + 2 * pad) - n) // 2
    rng = np.random.default_rng(n)
    dn = (0.02 * rng.standard_normal((slices, n, n))).astype(np.float32)
    ab = rng.uniform(0, 0.01, (slices, n, n)).astype(np.float32)
    u = _crand(rng, (n, n))
    bar = BAR * (1 + slices)
    ref = O.multislice_thick_sample(O.field_build(u, 0.15, 0.532), ab, dn, 1.33, 0.3, pad, NA=0.9).u
    f = _field(u, dx=0.15)
    d = to_cuda(dn).requires_grad_(True)
    out = cf.multislice_thick_sample(f, to_cuda(ab), d, 1.33, 0.3, pad, NA=0.9)
    assert O.rel_l2(out.u.detach().cpu().numpy(), np.asarray(ref).reshape(n, n)) < bar
    g = to_cuda(_crand(rng, (n, n)))
    (g0,) = torch.autograd.grad(out.u, d, g)
    d1 = to_cuda(dn).requires_grad_(True)
    (g1,) = torch.autograd.grad(cf.multislice_thick_sample(f, to_cuda(ab), d1, 1.33, 0.3, pad, NA=0.9, checkpoint_every=1).u, d1, g)
    assert torch.equal(g0, g1)
    # dL/d dn of the FP64 recursion, along one direction
    if pad == 0:
        w = rng.standard_normal(dn.shape).astype(np.float32)
        h = 1e-3
        gc = g.cpu().numpy().astype(np.complex128)
        L = [np.sum((gc.conj() * np.asarray(O.multislice_thick_sample(O.field_build(u, 0.15, 0.532), ab, dn + s * h * w, 1.33,
                                                                     0.3, 0, NA=0.9).u).reshape(n, n)).real) for s in (1, -1)]
        got = float(np.sum(g0.cpu().numpy().astype(np.float64) * w))
        assert abs(got - (L[0] - L[1]) / (2 * h)) < 1e-4 * np.linalg.norm(w) * float(torch.linalg.vector_norm(g0)) / np.sqrt(w.size) + 1e-2 * abs(got)


@pytest.mark.parametrize("n", [128, 160, 192, 224, 256, 320, 384, 448, 512])
@pytest.mark.parametrize("axis", [0, 1])
def test_mbs_strided_passes(n, axis):
    """One update of the modified Born series with one long strided axis (x: three components and the k-space
    operator; y), ragged tiles (20 columns) against the FP64 restatement: six transforms and the operator's
    reciprocals, eight FP32 roundings of the state."""
    import torch

    from chromatix_b200.experimental import mbs

    shape = (n, 16, 20) if axis == 0 else (16, n, 20)
    rng = np.random.default_rng(n)
    k0, sp = 2 * np.pi / 0.5, 0.1
    eps = 1.0 + 0.3 * rng.uniform(size=shape) + 0.02j * rng.uniform(size=shape)
    src = _crand(rng, shape + (3,))
    op = O.MBSOperator(eps.astype(np.complex64).astype(np.complex128), sp, k0, src.astype(np.complex128))
    sample = mbs.Sample(to_cuda(eps.astype(np.complex64)), sp)
    source = mbs.Source(torch.zeros(shape + (3,), dtype=torch.complex64, device="cuda"), k0)
    source.field = to_cuda(src)
    E = mbs.solve(sample, source, maxiter=1, tol=0.0, shift=op.bias, scale=op.scale).cpu().numpy()
    assert O.rel_l2(E, op.step(op.prec_y) * op.num_scale) < 2 * BAR


@pytest.mark.parametrize("ny,nx,pad,batch", [(2048, 2560, (0, 0), 1), (2048, 2560, (256, 0), 1), (640, 896, (0, 0), 10),
                                             (4096, 640, (0, 0), 2)])
def test_spectra_by_tile(ny, nx, pad, batch):
    """Spectra too large for half of the L2 are stored by tiles of eight columns: against the same field in batches
    that are stored by row, bit by bit (the arithmetic is the same)."""
    import torch

    import chromatix_b200.functional as cf

    rng = np.random.default_rng(ny + nx)
    u = _crand(rng, (batch, ny, nx))
    H = _crand(rng, (ny, nx))
    f = _field(u)
    big = cf.transfer_propagate(f, 30.0, 1.33, pad, mode="same").u
    if batch > 2:
        small = [cf.transfer_propagate(_field(u[b:b + 1]), 30.0, 1.33, pad, mode="same").u for b in range(batch)]
        assert torch.equal(big, torch.cat(small))
    ref = np.fft.ifft2(np.fft.fft2(u.astype(np.complex128)) * H)
    assert O.rel_l2(cf.kernel_propagate(f, to_cuda(H)).u.cpu().numpy(), ref) < BAR
    fy, fx = np.fft.fftfreq(ny + 2 * pad[0], 0.3), np.fft.fftfreq(nx + 2 * pad[1], 0.3)
    P = np.exp(-1j * np.pi * 0.532 * 30.0 / 1.33 * (fy[:, None] ** 2 + fx[None, :] ** 2))
    v = np.pad(u.astype(np.complex128), [(0, 0), (pad[0], pad[0]), (pad[1], pad[1])])
    out = np.fft.ifft2(np.fft.fft2(v) * P)[:, pad[0]:pad[0] + ny, pad[1]:pad[1] + nx]
    assert O.rel_l2(big.cpu().numpy(), out) < BAR


@pytest.mark.parametrize("n,m", [(64, 65), (65, 64), (100, 61), (129, 96), (300, 213), (513, 512), (700, 1349),
                                 (2000, 561), (2047, 2050), (4096, 4096)])
def test_chirp_z_pairs(n, m):
    """n + m - 1 at and beside a transform length, along contiguous rows (an odd number of them: half a pair) and along
    strided columns (odd and even numbers, a ragged last tile), against the sums in FP64.  Three FP32 transforms, three
    factors in 32 bits and the filter's spectrum: within the propagation's tolerance."""
    from chromatix_b200.utils.czt import czt

    rng = np.random.default_rng(n + m)
    a, w = np.exp(0.21j), np.exp(-1.7j / max(n, m))
    j, k = np.arange(n), np.arange(m)
    D = np.exp(1j * (np.angle(w) * np.outer(k, j) - np.angle(a) * j))
    for shape, axis in (((3, n), -1), ((2, n, 5), 1), ((n, 18), 0)):
        x = _crand(rng, shape)
        out = czt(to_cuda(x), m, a, w, axis=axis).cpu().numpy()
        ref = np.moveaxis(np.moveaxis(x.astype(np.complex128), axis, -1) @ D.T, -1, axis)
        assert O.rel_l2(out, ref) < BAR, shape


@pytest.mark.parametrize("batch,ny,nx,wv", [(1, 5, 7, 1), (3, 6, 10, 1), (4, 33, 31, 2), (17, 64, 64, 3)])
def test_phase_factor_over_a_batch(batch, ny, nx, wv):
    """One phase map for every field of a batch and one map per field, one and several wavelengths, odd and even row
    lengths.  FP32 sin / cos of arguments below 2 pi and one product: 4e-7."""
    import chromatix_b200.functional as cf

    rng = np.random.default_rng(batch + nx)
    lam = np.array([0.5, 0.45, 0.6][:wv]) if wv > 1 else 0.5
    u = _crand(rng, (batch, ny, nx) + ((wv,) if wv > 1 else ()))
    for shape in ((ny, nx), (batch, ny, nx)):
        ph = rng.uniform(-3, 3, shape).astype(np.float32)
        f = _field(u, lam=lam)
        out = cf.phase_change(f, to_cuda(ph)).u.cpu().numpy()
        p = ph.astype(np.float64)
        if wv > 1:
            p = p[..., None] * f.spectrum.spectral_modulation
        assert O.rel_l2(out, u * np.exp(1j * p)) < 4e-7


@pytest.mark.parametrize("shape", [(45, 75), (81, 99)])
def test_lengths_without_a_pass(shape):
    """Padded lengths with no fused pass: the planned route (no gradient asked for) against the route through autograd
    and against FP64; chirp-Z transforms instead of FFTs, twice the propagation's tolerance."""
    import torch

    import chromatix_b200.functional as cf

    rng = np.random.default_rng(shape[0])
    u = _crand(rng, (2,) + shape)
    f, g = _field(u), _field(u)
    g.u.requires_grad_(True)
    out = cf.asm_propagate(f, 25.0, 1.33, 6, mode="same").u
    grad = cf.asm_propagate(g, 25.0, 1.33, 6, mode="same").u.detach()
    assert torch.allclose(out, grad, rtol=0, atol=1e-5 * float(grad.abs().max()))
    for b in range(2):
        ref = O.asm_propagate(O.field_build(u[b], 0.3, 0.532), 25.0, 1.33, 6, mode="same").u
        assert O.rel_l2(out[b].cpu().numpy(), np.asarray(ref).reshape(shape)) < 2 * BAR
