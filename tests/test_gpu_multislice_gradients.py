"""GPU: the multislice adjoint with and without a second stream for its
recomputation."""

import ctypes

import numpy as np
import pytest

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
