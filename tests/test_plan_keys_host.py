"""Plan caches key a call by the values of its parameters (no GPU: the launch
is replaced by a recorder of the plan that it is given).

Every form in which a tilt, a shift or a spacing can be given leads to the plan
of its value, also after the caller has changed the value in place; forms that
only hash by identity, or not at all, are served like the others.
"""

import types

import numpy as np
import pytest
import torch

from chromatix_b200.core.field import ScalarField
from chromatix_b200.core.spectrum import Spectrum
from chromatix_b200.functional import propagation as P


def _field(shape=(16, 24), dx=0.3, lam=0.532):
    return ScalarField(torch.ones(shape, dtype=torch.complex64), dx, 0.0, Spectrum.build(lam))


@pytest.fixture
def launched(monkeypatch):
    """Descriptors and plane tables of the propagations launched, newest last."""
    seen = []

    def launch(plan, u):
        seen.append(types.SimpleNamespace(desc=plan.desc, planes=plan.planes))
        return torch.zeros(plan.out_shape, dtype=torch.complex64)

    def run_general(self, field):
        seen.append(types.SimpleNamespace(desc=self.h_desc, planes=self.planes))
        return torch.zeros(field.u.shape, dtype=torch.complex64)

    monkeypatch.setattr(P.nat, "require_cuda", lambda *a: None)
    monkeypatch.setattr(P, "_launch_prop2d", launch)
    monkeypatch.setattr(P._GeneralPlan, "run", run_general)
    monkeypatch.setattr(P, "_HOST_PLANS", type(P._HOST_PLANS)())
    return seen


FORMS = {
    "floats": lambda a, b: (a, b),
    "list": lambda a, b: [a, b],
    "array": lambda a, b: np.array([a, b]),
    "numpy scalars": lambda a, b: (np.float64(a), np.float64(b)),
    "0-d arrays": lambda a, b: (np.array(a), np.array(b)),
    "one-element arrays": lambda a, b: (np.array([a]), np.array([b])),
    "0-d tensors": lambda a, b: (torch.tensor(a, dtype=torch.float64), torch.tensor(b, dtype=torch.float64)),
    "tensor": lambda a, b: torch.tensor([a, b], dtype=torch.float64),
    "nested": lambda a, b: ((a, b),),
}


# 13 x 17: lengths without a fused pass (the route with its own plan)
@pytest.mark.parametrize("shape", [(16, 24), (13, 17)])
@pytest.mark.parametrize("form", FORMS)
def test_tilt_in_every_form(launched, shape, form):
    f = _field(shape)
    for v in ((0.25, -0.5), (0.125, 0.75), (0.25, -0.5)):
        P.transfer_propagate(f, 20.0, 1.33, 0, kykx=FORMS[form](*v))
        assert (launched[-1].desc.ky0, launched[-1].desc.kx0) == v


@pytest.mark.parametrize("shape", [(16, 24), (13, 17)])
@pytest.mark.parametrize("form", [k for k in FORMS if k not in ("one-element arrays", "nested")])
def test_shift_in_every_form(launched, shape, form):
    f = _field(shape)
    for v in ((0.25, -0.5), (0.125, 0.75), (0.25, -0.5)):
        P.asm_propagate(f, 20.0, 1.33, 0, shift_yx=FORMS[form](*v))
        p = launched[-1].planes[0]
        assert (p["shift_y"], p["shift_x"]) == v


@pytest.mark.parametrize("shape", [(16, 24), (13, 17)])
@pytest.mark.parametrize("make", [lambda: torch.tensor(0.25, dtype=torch.float64), lambda: np.array(0.25)])
def test_parameters_changed_in_place(launched, shape, make):
    f = _field(shape)
    t = make()
    for want in (0.25, 1.25, 2.25):
        P.asm_propagate(f, 20.0, 1.33, 0, kykx=(t, t), shift_yx=(t, 0.0))
        assert (launched[-1].desc.ky0, launched[-1].desc.kx0) == (want, want)
        assert launched[-1].planes[0]["shift_y"] == want
        t += 1


def test_spectrum_and_spacing_by_value(launched):
    for dx in (0.3, 0.6):
        for lam in (0.5, 0.6):
            P.transfer_propagate(_field(dx=dx, lam=lam), 20.0, 1.33, 0)
            p = launched[-1].planes[0]
            assert (p["dy"], p["wavelength"]) == (dx, lam)
