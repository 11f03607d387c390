"""The optical FFT's plan cache keys a call by the values of its parameters (no
GPU: the launch is replaced by a recorder of the plan that it is given)."""

import numpy as np
import pytest
import torch

from chromatix_b200.core.field import ChromaticScalarField, ScalarField
from chromatix_b200.core.spectrum import Spectrum
from chromatix_b200.functional import convenience as C
from chromatix_b200.functional import lenses


def _field(lam=0.532):
    spec = Spectrum.build(lam)
    u = torch.ones((16, 24) + ((spec.size,) if spec.size > 1 else ()), dtype=torch.complex64)
    return (ChromaticScalarField if spec.size > 1 else ScalarField)(u, 0.3, 0.0, spec)


@pytest.fixture
def planes(monkeypatch):
    """Plane tables of the optical FFTs launched, newest last."""
    seen = []

    def launch(plan, u):
        seen.append(plan.planes)
        return torch.zeros(plan.out_shape, dtype=torch.complex64)

    monkeypatch.setattr(C.nat, "require_cuda", lambda *a: None)
    monkeypatch.setattr(C, "_launch_optfft", launch)
    monkeypatch.setattr(C, "_OPT_PLANS", type(C._OPT_PLANS)())
    return seen


FORMS = {
    "float": float,
    "int": int,
    "numpy scalar": np.float64,
    "0-d array": np.array,
    "one-element array": lambda v: np.array([v]),
    "0-d tensor": lambda v: torch.tensor(v, dtype=torch.float64),
}


@pytest.mark.filterwarnings("ignore::DeprecationWarning")
@pytest.mark.parametrize("lens,form", [(k, m) for k in ("ff", "df") for m in FORMS if (k, m) != ("df", "0-d tensor")])
def test_lens_parameters_in_every_form(planes, lens, form):
    make = FORMS[form]
    for f, n, NA in ((100.0, 1.0, 2.0), (200.0, 2.0, 1.0), (100.0, 1.0, 3.0), (100.0, 1.0, 2.0)):
        if lens == "ff":
            lenses.ff_lens(_field(), make(f), make(n), make(NA))
        else:
            lenses.df_lens(_field(), make(50.0), make(f), make(n), make(NA))
        D = 2 * f * NA / n
        assert planes[-1][0]["pupil_r2"] == (D / 2) ** 2
        assert planes[-1][0]["dy_out"] == pytest.approx(0.532 * f / n / (16 * 0.3), rel=1e-12)


@pytest.mark.parametrize("make", [lambda: torch.tensor(2.0, dtype=torch.float64), lambda: np.array(2.0)])
def test_aperture_changed_in_place(planes, make):
    NA = make()
    for want in (2.0, 3.0, 4.0):
        lenses.ff_lens(_field(), 100.0, 1.0, NA)
        assert planes[-1][0]["pupil_r2"] == (100.0 * want) ** 2
        NA += 1


def test_factors_by_value_not_by_bytes(planes):
    """Equal bytes of unequal types or shapes are different factors."""
    f = _field(np.array([0.5, 0.6]))
    one = np.array([1.0, 0.5])
    for post in (one, one.view(np.int64), one.view(np.complex128)[0]):
        C.run_optfft(f, 100.0, 1.0, post=post)
        want = np.broadcast_to(np.asarray(post, dtype=np.complex128), (2,))
        np.testing.assert_array_equal(planes[-1]["post_re"] + 1j * planes[-1]["post_im"], want)
    for chirp in (one, one.view(np.int64)):
        C.run_optfft(f, 100.0, 1.0, chirp_in=chirp)
        np.testing.assert_array_equal(planes[-1]["chirp_in"], chirp.astype(np.float64))


@pytest.mark.parametrize("make", [lambda: torch.tensor(2), lambda: np.array(2)])
def test_padding_changed_in_place(planes, make):
    from chromatix_b200.functional import propagation as P

    p = make()
    for want in (2, 3, 4):
        out = P.transform_propagate(_field(), 100.0, 1.0, (p, p))
        assert tuple(out.u.shape) == (16, 24)
        # the spacing of the padded grid
        assert planes[-1][0]["dy_out"] == pytest.approx(0.532 * 100.0 / ((16 + 2 * want) * 0.3), rel=1e-12)
        p += 1
