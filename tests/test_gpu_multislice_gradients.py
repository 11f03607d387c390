"""GPU: the multislice adjoint, with and without a second stream for its
recomputation, and every gradient against an FP64 restatement of the recursion.

Bars: an FP32 transform of length N rounds with a relative L2 error of about
0.5 eps sqrt(log2 N) <= 1e-7; a slice's step is four of them and a product,
2.5e-7 in squares.  u_D passes D slices and the defocus, the adjoint as many
again, and a gradient is the product of a field of each: at most 2 (D + 2)
steps added without cancellation, 5e-7 (D + 2).  The bar is twice that.  The
FP32 transmittances round like one more product.
"""

import ctypes

import numpy as np
import pytest

from oracle import chromatix_oracle as O

pytestmark = pytest.mark.gpu

LAM, DZ, N_MED, DX = 0.532, 0.2, 1.33, 0.1


def _rng_case(n, pad, D, seed):
    ny, nx = n
    rng = np.random.default_rng(seed)
    u = (rng.standard_normal((ny, nx)) + 1j * rng.standard_normal((ny, nx))).astype(np.complex64)
    g = (rng.standard_normal((ny, nx)) + 1j * rng.standard_normal((ny, nx))).astype(np.complex64)
    dn = (0.02 * rng.standard_normal((D, ny, nx))).astype(np.float32)
    ab = rng.uniform(0, 0.01, (D, ny, nx)).astype(np.float32)
    return u, g, dn, ab


def _asm(shape, z):
    f = O.field_build(np.ones(shape, dtype=np.complex128), DX, LAM)
    return np.asarray(O.compute_asm_propagator(f, z, N_MED)).reshape(shape)


def _fp64_gradients(u, g, dn, ab, pad, NA):
    """u_0 = pad u, u_{i+1} = t_i P u_i, out = crop Q u_D; the adjoint of each step in reverse."""
    D, ny, nx = dn.shape
    P = [(pad, pad), (pad, pad)]
    v = np.pad(u.astype(np.complex128), P)
    H, Q = _asm(v.shape, DZ), _asm(v.shape, -DZ * D / 2)
    fy, fx = np.fft.fftfreq(v.shape[0], DX), np.fft.fftfreq(v.shape[1], DX)
    Q = Q * (fy[:, None] ** 2 + fx[None, :] ** 2 <= (NA / LAM) ** 2)
    k = 2 * np.pi * DZ / LAM
    t = [np.pad(np.exp(1j * k * (dn[i].astype(np.float64) + 1j * ab[i])), P, constant_values=1.0) for i in range(D)]
    fields = []
    for i in range(D):
        v = t[i] * np.fft.ifft2(H * np.fft.fft2(v))
        fields.append(v)
    out = np.fft.ifft2(Q * np.fft.fft2(v))[pad:pad + ny, pad:pad + nx]
    w = np.fft.ifft2(Q.conj() * np.fft.fft2(np.pad(g.astype(np.complex128), P)))
    gdn, gab = np.empty(dn.shape), np.empty(dn.shape)
    for i in reversed(range(D)):
        p = (w * fields[i].conj())[pad:pad + ny, pad:pad + nx]
        gdn[i], gab[i] = k * p.imag, -k * p.real
        w = np.fft.ifft2(H.conj() * np.fft.fft2(t[i].conj() * w))
    return out, gdn, gab, w[pad:pad + ny, pad:pad + nx]


# Padded sides with a pair plan (the last: 64 rows without).  Odd paddings: a pair of rows straddles the edge of the
# data.  Widths that 4 does not divide: rows read element by element, records by the bulk copy's fallback.
@pytest.mark.parametrize("n,pad,D", [((128, 128), 0, 4), ((130, 130), 15, 4), ((98, 98), 15, 5), ((226, 226), 15, 3),
                                     ((102, 166), 13, 3), ((70, 134), 29, 3), ((256, 128), 0, 6), ((62, 126), 1, 4)])
@pytest.mark.parametrize("K", [0, 1, 2])
def test_every_gradient_against_fp64(n, pad, D, K):
    import torch

    import chromatix_b200 as cx
    import chromatix_b200.functional as cf

    u, g, dn, ab = _rng_case(n, pad, D, seed=n[0] + pad)
    out64, gdn64, gab64, gu64 = _fp64_gradients(u, g, dn, ab, pad, 0.9)
    # the restatement's forward is the oracle's
    ref = O.multislice_thick_sample(O.field_build(u, DX, LAM), ab, dn, N_MED, DZ, pad, NA=0.9).u
    assert O.rel_l2(out64, np.asarray(ref).reshape(n)) < 1e-9
    ut, dnt, abt = (torch.as_tensor(x, device="cuda").requires_grad_(True) for x in (u, dn, ab))
    f = cx.ScalarField(ut, DX, 0.0, cx.MonoSpectrum(LAM))
    out = cf.multislice_thick_sample(f, abt, dnt, N_MED, DZ, pad, NA=0.9, checkpoint_every=K).u
    gu, gdn, gab = torch.autograd.grad(out, (ut, dnt, abt), torch.as_tensor(g, device="cuda"))
    bar = 1e-6 * (D + 2)
    assert O.rel_l2(out.detach().cpu().numpy(), out64) < bar
    for i in range(D):
        assert O.rel_l2(gdn[i].cpu().numpy(), gdn64[i]) < bar, i
        assert O.rel_l2(gab[i].cpu().numpy(), gab64[i]) < bar, i
    assert O.rel_l2(gu.cpu().numpy(), gu64) < bar
    # no element is off by more than a row's or column's misplacement would make it
    for a, b in ((gdn, gdn64), (gab, gab64)):
        assert np.max(np.abs(a.cpu().numpy() - b)) < 8 * bar * np.sqrt(np.mean(b ** 2)) * np.sqrt(np.log(b.size))


@pytest.mark.parametrize("n,pad,D,K", [((128, 128), 0, 24, 5), ((130, 130), 15, 9, 2), ((512, 512), 0, 12, 3),
                                       ((1024, 1024), 0, 10, 4), ((128, 128), 0, 7, 1), ((64, 64), 0, 9, 4)])
def test_one_stream_gives_the_same_bits(n, pad, D, K):
    """The recomputation on the caller's stream alone: the first adjoint pass of
    a segment follows the pass that wrote the record which it reads."""
    import torch

    from chromatix_b200 import _native as nat
    from chromatix_b200.functional import samples as S

    u, g, dn, ab = (torch.as_tensor(x, device="cuda") for x in _rng_case(n, pad, D, seed=3))
    d = S.cx_ms_desc()
    d.ny, d.nx, d.pad, d.n_slices, d.checkpoint_every = *n, pad, D, K
    d.n_medium, d.wavelength, d.dy, d.dx, d.dz = N_MED, LAM, DX, DX, DZ
    d.reverse_distance, d.NA = DZ * D / 2, 0.9
    L = S._ms_lib()
    V = ctypes.c_void_p
    L.cx_multislice_backward_one_stream.restype = ctypes.c_int32
    L.cx_multislice_backward_one_stream.argtypes = [ctypes.POINTER(S.cx_ms_desc)] + [V] * 8 + [nat.c_size_t, V]
    _, ck = S._ms_forward(d, u, dn, ab, want_ckpt=True)
    want = S._ms_backward(d, dn, ab, ck, g, need_u=True)
    size = nat.c_size_t(0)
    nat.check(L.cx_multislice_workspace_size(d, 1, size))
    ws = nat.workspace(size.value, u.device)
    got = (torch.empty_like(dn), torch.empty_like(ab), torch.empty_like(u))
    for _ in range(4):
        for t in got:
            t.zero_()
        nat.check(L.cx_multislice_backward_one_stream(d, nat.ptr(dn), nat.ptr(ab), nat.ptr(ck), nat.ptr(g),
                                                      *(nat.ptr(t) for t in got), nat.ptr(ws), size.value,
                                                      nat.stream_handle(u.device)))
        for a, b in zip(got, want):
            assert torch.equal(a, b)
