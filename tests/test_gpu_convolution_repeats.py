"""GPU: the plane sum of the convolution is the same bits from call to call.

Few columns and many planes: several CTAs sum the planes of one column, and
the order in which they finish must not decide the rounding.  Values against
FP64: four FP32 transforms and products, 1.3e-6 as for the other tests of
these passes.
"""

import numpy as np
import pytest

from oracle import chromatix_oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("planes,h,w", [(3, 64, 64), (16, 200, 200), (33, 70, 130), (64, 128, 128), (64, 256, 256),
                                        (7, 512, 512), (48, 700, 130), (48, 130, 700), (40, 768, 768), (2, 96, 128),
                                        (300, 64, 128)])
def test_plane_sum_repeats_bit_for_bit(planes, h, w):
    import torch

    from chromatix_b200.ops import fourier_convolution

    rng = np.random.default_rng(planes + w)
    a = rng.uniform(size=(planes, h, w)).astype(np.float32)
    k = rng.uniform(size=(planes, h, w)).astype(np.float32) ** 4
    at, kt = torch.as_tensor(a, device="cuda"), torch.as_tensor(k, device="cuda")
    out = fourier_convolution(at, kt, reduce=True)
    F = sum(np.fft.rfft2(x.astype(np.float64), (2 * h, 2 * w)) * np.fft.rfft2(y.astype(np.float64), (2 * h, 2 * w))
            for x, y in zip(a, k))
    y0, x0 = (h - 1) // 2, (w - 1) // 2
    ref = np.fft.irfft2(F, (2 * h, 2 * w))[y0:y0 + h, x0:x0 + w]
    assert O.rel_l2(out.cpu().numpy(), ref) < 1.3e-6
    for _ in range(12):
        assert torch.equal(fourier_convolution(at, kt, reduce=True), out)
