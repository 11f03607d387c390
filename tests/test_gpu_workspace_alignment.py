"""GPU: workspaces on an 8-byte boundary (what the planes and fields in them
need) give the results of 256-byte aligned ones, bit for bit, also where the
passes move 16 bytes at a time; and nothing is written past their end."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


class _Shifted:
    """Workspaces shifted by ``off`` bytes inside a larger block, whose rest is watched."""

    def __init__(self, off):
        self.off, self.blocks = off, []

    def __call__(self, nbytes, device):
        import torch

        n = max(int(nbytes), 256)
        block = torch.full((n + 512,), 0xA5, dtype=torch.uint8, device=device)
        self.blocks.append((block, n))
        return block[self.off:self.off + n]

    def intact(self):
        return all(bool((b[:self.off] == 0xA5).all()) and bool((b[self.off + n:] == 0xA5).all()) for b, n in self.blocks)


def _calls():
    import torch

    import chromatix_b200 as cx
    import chromatix_b200.functional as cf
    from chromatix_b200.ops import fourier_convolution

    rng = np.random.default_rng(2)

    def f32(*s):
        return torch.as_tensor(rng.uniform(size=s).astype(np.float32), device="cuda")

    for planes, h, w in ((3, 65, 70), (2, 80, 131), (40, 64, 128), (5, 20, 30)):
        a, k = f32(planes, h, w), f32(planes, h, w)
        yield fourier_convolution(a, k)
        yield fourier_convolution(a, k, reduce=True)
    for n in ((128, 160), (96, 128), (192, 5), (64, 48)):
        f = cf.objective_point_source(n, 0.3, 0.532, np.array([-2.0, 0.5]), 100.0, 1.33, 0.4, device="cuda")
        yield cf.ff_lens(cf.phase_change(f, f32(*n)), 200.0, 1.33).intensity
    u = torch.complex(f32(3, 128, 160), f32(3, 128, 160))
    g = cx.ScalarField(u, 0.3, 0.0, cx.MonoSpectrum(0.532))
    yield cf.asm_propagate(g, 20.0, 1.33, 32, mode="same").u
    yield cf.asm_propagate(g, 20.0, 1.33, 3, mode="same").u
    yield cf.ff_lens(g, 200.0, 1.33).u


@pytest.mark.parametrize("off", [8, 16, 24])
def test_shifted_workspaces(monkeypatch, off):
    import torch

    from chromatix_b200 import _native as nat

    want = list(_calls())
    ws = _Shifted(off)
    monkeypatch.setattr(nat, "workspace", ws)
    for i, (a, b) in enumerate(zip(_calls(), want)):
        assert torch.equal(a, b), i
    assert ws.blocks and ws.intact()
