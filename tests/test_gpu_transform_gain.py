"""GPU: the mean gain of the transforms on pairs of vectors.

A propagation over no distance is four transforms and a multiplication by one:
its output is the input, but for rounding.  The part of the error that all
points share, Re <u, out - u> / <u, u>, is set by the twiddle factors' and the
butterflies' rounded constants: at most 2.5e-8 for each transform (the gain of
the plan as a linear map, evaluated in FP64 from its rounded constants), 1e-7
for four, and the rounding of the scale 1 / N, 6e-8 where N is no power of two.
A white field also has its random errors, 3e-7 / sqrt(points) here; a constant
one passes the factor one alone.
"""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ny,nx", [(128, 128), (256, 256), (512, 512), (1024, 1024), (2048, 2048), (384, 768),
                                   (1536, 896), (640, 1280), (3072, 192), (1792, 2560), (4096, 448), (8192, 256)])
@pytest.mark.parametrize("white", [True, False])
def test_round_trip(ny, nx, white):
    import torch

    import chromatix_b200 as cx
    import chromatix_b200.functional as cf

    rng = np.random.default_rng(ny + nx)
    shape = (4, ny, nx)
    u = np.ones(shape, dtype=np.complex64)
    if white:
        u = (rng.standard_normal(shape) + 1j * rng.standard_normal(shape)).astype(np.complex64)
    out = cf.asm_propagate(cx.ScalarField(torch.as_tensor(u, device="cuda"), 0.3, 0.0, cx.MonoSpectrum(0.532)), 0.0, 1.33, 0).u.cpu().numpy()
    d = (out.astype(np.complex128) - u).ravel()
    v = u.astype(np.complex128).ravel()
    n = np.vdot(v, v).real
    scale = 0.0 if (ny & (ny - 1)) == 0 and (nx & (nx - 1)) == 0 else 6e-8
    assert abs(np.vdot(v, d).real) / n < 1e-7 + scale
    # four transforms' random errors, 0.35 eps sqrt(log2 N) each and none at all for the constant field's zeros
    assert np.linalg.norm(d) / np.sqrt(n) < 2 * 0.35 * 1.2e-7 * np.sqrt(2 * np.log2(ny * nx)) + 1e-7 + scale
