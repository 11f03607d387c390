"""The caches of plans and device tables with several threads (no GPU: launches
and uploads are replaced by recorders).

More keys than a cache holds, so that entries are evicted by one thread while
another has just found them: no call may fail, and each gets its own plan.
"""

import sys
import threading

import numpy as np
import pytest
import torch

from chromatix_b200 import _native as nat
from chromatix_b200.core.field import ScalarField
from chromatix_b200.core.spectrum import Spectrum
from chromatix_b200.functional import convenience as C
from chromatix_b200.functional import lenses
from chromatix_b200.functional import propagation as P

N_THREADS, KEYS, ROUNDS = 8, 200, 3


@pytest.fixture
def busy_switching():
    old = sys.getswitchinterval()
    sys.setswitchinterval(1e-6)
    yield
    sys.setswitchinterval(old)


def _field():
    return ScalarField(torch.ones((4, 4), dtype=torch.complex64), 0.3, 0.0, Spectrum.build(0.5))


def _run(call):
    """``call(k)`` for every key from every thread; the first exception is raised here."""
    errors = []

    def work(start):
        try:
            for i in range(KEYS * ROUNDS):
                call((start + i) % KEYS)
        except BaseException as e:  # noqa: BLE001
            errors.append(e)

    threads = [threading.Thread(target=work, args=(KEYS * t // N_THREADS,)) for t in range(N_THREADS)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    if errors:
        raise errors[0]


class _EvictedOnceFound(type(P._HOST_PLANS)):
    """A cache in which another thread evicts each entry as soon as it has been looked up."""

    def get(self, key):
        hit = super().get(key)
        if hit is not None:
            self.clear()
        return hit


def test_propagation_plans(monkeypatch, busy_switching):
    f = _field()
    monkeypatch.setattr(P.nat, "require_cuda", lambda *a: None)
    monkeypatch.setattr(P, "_launch_prop2d", lambda plan, u: torch.full((1,), plan.planes[0]["z"]))
    for cache in (type(P._HOST_PLANS)(), _EvictedOnceFound()):
        monkeypatch.setattr(P, "_HOST_PLANS", cache)

        def call(k):
            assert float(P._run_prop2d(f, nat.CX_KERNEL_TRANSFER, np.array([1.0 + k]), (), 1.33, 0)) == 1.0 + k

        call(0), call(0)
        _run(call)


def test_optical_fft_plans(monkeypatch, busy_switching):
    f = _field()
    monkeypatch.setattr(C.nat, "require_cuda", lambda *a: None)
    monkeypatch.setattr(C, "_launch_optfft", lambda plan, u: torch.tensor(plan.planes[0]["dy_out"]))
    for cache in (type(C._OPT_PLANS)(), _EvictedOnceFound()):
        monkeypatch.setattr(C, "_OPT_PLANS", cache)

        def call(k):
            u, du = C.run_optfft(f, 1.0 + k, 1.0)
            assert float(u) == du[0, 0] == pytest.approx(0.5 * (1.0 + k) / (4 * 0.3), rel=1e-12)

        call(0), call(0)
        _run(call)


class _Event:
    def record(self, stream):
        pass

    def query(self):
        return True


def test_device_tables(monkeypatch, busy_switching):
    fake = type("torch", (), {"cuda": type("cuda", (), {
        "Event": _Event, "is_current_stream_capturing": staticmethod(lambda: False),
        "current_stream": staticmethod(lambda device=None: None)})})
    monkeypatch.setattr(nat, "torch_mod", lambda: fake)
    monkeypatch.setattr(nat, "device_index", lambda device=None: 0)
    monkeypatch.setattr(nat, "stream_handle", lambda device=None: 7)
    monkeypatch.setattr(nat, "upload", lambda arr, device: arr.copy())

    def call(k):
        assert nat.constant(np.array([float(k)]), None)[0] == k

    for cache in (type(nat._TABLES)(), _EvictedOnceFound()):
        monkeypatch.setattr(nat, "_TABLES", cache)
        call(0), call(0)
        _run(call)
