"""A constant first used in inference mode serves a training step afterwards
(no GPU: the copy to the device stays on the host)."""

import numpy as np
import pytest
import torch

from chromatix_b200 import _native as nat


@pytest.fixture
def host(monkeypatch):
    class Event:
        def record(self, stream=None):
            pass

    monkeypatch.setattr(torch.cuda, "Event", Event)
    monkeypatch.setattr(torch.cuda, "current_stream", lambda device=None: None)
    monkeypatch.setattr(nat, "device_index", lambda device=None: 0)
    monkeypatch.setattr(nat, "stream_handle", lambda device=None: 0)
    monkeypatch.setattr(nat, "_pinned", lambda arr: torch.from_numpy(np.array(arr)))
    monkeypatch.setattr(nat, "_CONSTANTS", nat.PlanCache())


class Scale(torch.autograd.Function):
    @staticmethod
    def forward(ctx, x, c):
        ctx.save_for_backward(c)
        return x * c

    @staticmethod
    def backward(ctx, g):
        (c,) = ctx.saved_tensors
        return g * c, None


def test_constant_of_an_evaluation_in_a_training_step(host):
    density = np.array([0.25, 0.75])
    with torch.inference_mode():
        kept = nat.constant(density, "cpu")
    assert nat.constant(density, "cpu") is kept
    x = torch.ones(2, dtype=torch.float64, requires_grad=True)
    Scale.apply(x, nat.constant(density, "cpu")).sum().backward()
    assert x.grad.tolist() == density.tolist()
