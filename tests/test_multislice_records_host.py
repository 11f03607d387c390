"""The slice fields that multislice gradients keep until their backward pass
(no GPU: the native calls are replaced by recorders of the checkpoint spacing).

By default a call keeps every slice's field; all calls that wait for their
backward pass together keep 4 GiB that way, the others a field every sqrt(D).
"""

import math

import pytest
import torch

from chromatix_b200.core.field import ScalarField
from chromatix_b200.core.spectrum import Spectrum
from chromatix_b200.functional import samples as S

LIMIT = 4 << 30
N, D = 2048, 60  # 61 planes of 32 MiB: two calls fit the limit, three do not
PLANE = 8 * N * N
ROOT = math.ceil(math.sqrt(D))


@pytest.fixture
def spacings(monkeypatch):
    """``checkpoint_every`` of the forward calls, oldest first."""
    seen = []

    def forward(d, u, dn, ab, want_ckpt):
        seen.append(d.checkpoint_every)
        return torch.zeros_like(u), torch.empty(1) if want_ckpt else None

    def backward(d, dn, ab, ck, g, need_u):
        return None, None, torch.zeros_like(g) if need_u else None

    monkeypatch.setattr(S, "_ms_forward", forward)
    monkeypatch.setattr(S, "_ms_backward", backward)
    monkeypatch.setattr(S, "_MS_FN", None)
    return seen


def _call(batch, requires_grad=True, **kw):
    u = torch.zeros((N, N), dtype=torch.complex64).expand((batch, N, N)).requires_grad_(requires_grad)
    f = ScalarField(u, 0.1, 0.0, Spectrum.build(0.532))
    dn = torch.empty((D, N, N))  # (never written: takes no memory)
    return S.multislice_thick_sample(f, dn, dn, 1.33, 0.2, 0, **kw).u


def _held(spacings):
    """Bytes of the fields kept by calls of these spacings (0: the library's own rule for one call)."""
    total = 0
    for K in spacings:
        K = min(K, D) if K > 0 else D
        segments = -(-D // K)
        total += (segments + D - (segments - 1) * K) * PLANE
    return total


def test_batch_shares_the_limit(spacings):
    out = _call(5)
    assert len(spacings) == 5
    assert _held(spacings) <= LIMIT + 5 * 2 * ROOT * PLANE
    assert spacings == [D, D, ROOT, ROOT, ROOT]
    del out


def test_calls_that_wait_for_their_backward_pass_share_the_limit(spacings):
    outs = [_call(1) for _ in range(4)]
    assert _held(spacings) <= LIMIT + 4 * 2 * ROOT * PLANE
    # a backward pass and a result that is dropped give their share back
    outs[0].real.sum().backward()
    outs.append(_call(1))
    assert spacings[-1] == D
    outs.append(_call(1))
    assert spacings[-1] == ROOT
    del outs[1]
    outs.append(_call(1))
    assert spacings[-1] == D


def test_a_training_loop_keeps_every_field(spacings):
    for _ in range(6):
        loss = _call(2).real.sum()
        loss.backward()
    assert spacings == [D] * 12


def test_without_gradients_nothing_is_kept(spacings):
    outs = [_call(2, requires_grad=False) for _ in range(3)] + [_call(2)]
    assert spacings[-2:] == [D, D]
    del outs


def test_an_explicit_spacing_is_as_asked(spacings):
    out = [_call(3, checkpoint_every=k) for k in (1, 7, D, D, 2 * D)]
    assert spacings == [k for k in (1, 7, D, D, 2 * D) for _ in range(3)]
    del out


def test_a_failed_call_gives_its_share_back(spacings, monkeypatch):
    good = S._ms_forward
    for _ in range(3):
        monkeypatch.setattr(S, "_ms_forward", lambda *a, **k: (_ for _ in ()).throw(RuntimeError("no memory")))
        with pytest.raises(RuntimeError, match="no memory"):
            _call(1)
    monkeypatch.setattr(S, "_ms_forward", good)
    out = _call(2)
    assert spacings == [D, D]
    del out
