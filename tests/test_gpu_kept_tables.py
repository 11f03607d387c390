"""GPU: kept device tables under capture and on several streams."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _field(u, lam, dx=0.3):
    import chromatix_b200 as cx
    from chromatix_b200.core.spectrum import Spectrum

    spec = Spectrum.build(lam)
    return (cx.ChromaticScalarField if spec.size > 1 else cx.ScalarField)(u, dx, 0.0, spec)


def _calls(u, ph, lam, z):
    import chromatix_b200.functional as cf

    f = _field(u, lam)
    yield cf.transfer_propagate(f, z, 1.33, 0).u
    yield cf.asm_propagate(f, z, 1.33, (5, 6), mode="same").u  # a length without a fused pass
    yield cf.ff_lens(f, z, 1.33).u
    yield cf.phase_change(f, ph).u
    yield f.intensity


def test_first_call_inside_a_capture():
    """Geometries, densities and factors that are new inside a capture: eager
    calls before the first replay do not read what the graph has yet to write,
    and every replay writes it again, also after the cache has turned over."""
    import torch

    from chromatix_b200 import _native as nat

    rng = np.random.default_rng(0)
    shape = (64, 96, 3)

    def rand():
        a = (rng.standard_normal(shape) + 1j * rng.standard_normal(shape)).astype(np.complex64)
        return torch.as_tensor(a, device="cuda")

    u, ph = rand(), torch.as_tensor(rng.uniform(-3, 3, shape[:2]).astype(np.float32), device="cuda")
    warm, lam = (np.array([0.5, 0.6, 0.7]), np.array([1.0, 2.0, 3.0])), (np.array([0.45, 0.55, 0.65]), np.array([3.0, 1.0, 5.0]))
    for _ in _calls(u, ph, warm, 30.0):
        pass
    side = torch.cuda.Stream()
    with torch.cuda.stream(side):
        for _ in _calls(u, ph, warm, 31.0):
            pass
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        out = list(_calls(u, ph, lam, 40.0))
    eager = [t.clone() for t in _calls(u, ph, lam, 40.0)]
    g.replay()
    for a, b in zip(out, eager):
        assert torch.equal(a, b)
    for k in range(300):
        nat.constant(np.array([float(k), 0.5]), u.device)
        d = nat.cx_ew_desc(n_batch=k + 1, ny=1, nx=1, n_wv=1, map_batched=0)
        nat.device_table(d, np.zeros(1, dtype=nat.PLANE_DTYPE), u.device, lambda desc: 0)
    for _ in range(3):
        u.copy_(rand())
        g.replay()
        for a, b in zip(out, _calls(u, ph, lam, 40.0)):
            assert torch.equal(a, b)


def test_eviction_while_another_stream_reads():
    """A constant uploaded on one stream, read late on another, evicted and its
    memory asked for again on the first."""
    import torch

    from chromatix_b200 import _native as nat

    torch.cuda.synchronize()
    a, b = torch.cuda.Stream(), torch.cuda.Stream()
    rng = np.random.default_rng(1)
    u = torch.as_tensor((rng.standard_normal((512, 512, 2)) + 0j).astype(np.complex64), device="cuda")
    lam = (np.array([0.41, 0.52]), np.array([0.3, 0.7]))
    busy = torch.empty((64 << 20,), device="cuda")
    with torch.cuda.stream(a):
        want = _field(u, lam).intensity
    torch.cuda.synchronize()
    with torch.cuda.stream(b):
        for _ in range(40):
            busy.add_(1.0)  # keeps the stream busy while the host goes on
        got = _field(u, lam).intensity
    with torch.cuda.stream(a):
        for k in range(300):
            nat.constant(np.array([float(k), 7.0]), u.device)
        junk = [torch.full((2,), 1e30, dtype=torch.float64, device="cuda") for _ in range(2000)]
    torch.cuda.synchronize()
    assert torch.equal(got, want)
    del junk
