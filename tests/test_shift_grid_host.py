"""shift_grid sets the origin to the same array for every form of the shift."""

import numpy as np
import pytest
import torch

from chromatix_b200.core.field import ScalarField, shift_grid
from chromatix_b200.core.spectrum import Spectrum


def _by_definition(origin, shift):
    s = np.atleast_1d(np.asarray(shift, dtype=np.float64))
    if s.size < 2:
        s = np.array([s[0], s[0]])
    if s.size != 2:
        raise AssertionError
    return np.zeros_like(np.asarray(origin, dtype=np.float64)) + s


@pytest.mark.parametrize("origin", [0.0, [0.0], [1.0, 2.0]])
@pytest.mark.parametrize("shift", [0.5, (0.5,), (0.5, -1.0), [0.5, -1.0], (1, 2), np.array([0.5, -1.0]),
                                   (np.array(0.5), np.array(-1.0)), (np.array([0.5]), np.array([-1.0])),
                                   (torch.tensor(0.5), torch.tensor(-1.0)), ([0.5], [-1.0]),
                                   ([0.5, 0.5], [-1.0, -1.0]), (0.5, -1.0, 2.0)])
def test_every_form(origin, shift):
    f = ScalarField(torch.ones((4, 6), dtype=torch.complex64), 0.3, np.asarray(origin), Spectrum.build(0.5))
    try:
        want = _by_definition(f.origin, shift)
    except AssertionError:
        with pytest.raises(AssertionError):
            shift_grid(f, shift)
        return
    got = np.asarray(shift_grid(f, shift).origin)
    assert got.dtype == np.float64
    np.testing.assert_array_equal(got, want)
    assert got.shape == want.shape
