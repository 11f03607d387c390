"""Device copies of plane tables and constants: which stream may use them, and
how long they live (no GPU: torch's CUDA calls are replaced by recorders)."""

import gc
import weakref

import numpy as np
import pytest

from chromatix_b200 import _native as nat


class Table:
    """A device tensor of the fake: remembers the streams it was recorded on."""

    def __init__(self, arr):
        self.arr, self.recorded = np.array(arr), []

    def record_stream(self, stream):
        self.recorded.append(stream.handle)


class Stream:
    def __init__(self, handle, log):
        self.handle, self.log = handle, log

    def wait_event(self, ev):
        self.log.append(("wait", self.handle, ev.recorded_on))


class Fake:
    """torch.cuda with one current stream that the test sets."""

    def __init__(self):
        self.handle, self.capturing, self.log = 1, False, []
        fake = self

        class Event:
            recorded_on = None

            def record(self, stream=None):
                assert not fake.capturing or stream.handle == fake.handle
                self.recorded_on = stream.handle

            def query(self):
                raise AssertionError("an event's query ends the capture that another thread has open")

        class cuda:
            pass

        cuda.Event = Event
        cuda.is_current_stream_capturing = staticmethod(lambda: fake.capturing)
        cuda.current_stream = staticmethod(lambda device=None: Stream(fake.handle, fake.log))
        self.cuda = cuda

    def is_in(self, handle, capturing=False):
        self.handle, self.capturing = handle, capturing


@pytest.fixture
def gpu(monkeypatch):
    fake = Fake()
    monkeypatch.setattr(nat, "torch_mod", lambda: fake)
    monkeypatch.setattr(nat, "device_index", lambda device=None: 0)
    monkeypatch.setattr(nat, "stream_handle", lambda device=None: fake.handle)
    monkeypatch.setattr(nat, "upload", lambda arr, device: Table(arr))
    monkeypatch.setattr(nat, "_CAPTURED", {})
    for name in ("_TABLES", "_CONSTANTS"):
        monkeypatch.setattr(nat, name, nat.PlanCache(128))
    return fake


def constant(v):
    return nat.constant(np.array([v], dtype=np.float64), "cuda:0")


def plane_table(v):
    d = nat.cx_ew_desc(n_batch=1, ny=1, nx=1, n_wv=1, map_batched=0)
    planes = np.zeros(1, dtype=nat.PLANE_DTYPE)
    planes["z"] = v
    return nat.device_table(d, planes, "cuda:0", lambda desc: 256)[1]


@pytest.mark.parametrize("make", [constant, plane_table])
def test_use_on_another_stream(gpu, make):
    """The first use on a stream other than the uploading one waits for the
    upload and tells the allocator of that stream; later uses do neither."""
    t = make(1.0)
    assert make(1.0) is t
    assert t.recorded == [] and gpu.log == []
    gpu.is_in(2)
    assert make(1.0) is t and make(1.0) is t
    assert t.recorded == [2] and gpu.log == [("wait", 2, 1)]
    gpu.is_in(3)
    assert make(1.0) is t
    gpu.is_in(2)
    assert make(1.0) is t
    gpu.is_in(1)
    assert make(1.0) is t
    assert t.recorded == [2, 3] and gpu.log == [("wait", 2, 1), ("wait", 3, 1)]


@pytest.mark.parametrize("make", [constant, plane_table])
def test_first_call_inside_a_capture(gpu, monkeypatch, make):
    """A table uploaded inside a capture holds its values only once the graph
    has run: later calls get their own, and what the graph copies from lives on."""
    hosts = []

    class Host:
        def __init__(self, arr):
            self.arr = np.array(arr)
            hosts.append(weakref.ref(self))

        def to(self, device, non_blocking=False):
            return Table(self.arr)

    monkeypatch.setattr(nat, "_pinned", Host, raising=False)
    gpu.is_in(5, capturing=True)
    t = make(3.0)
    gpu.is_in(5)
    eager = make(3.0)
    assert eager is not t and make(3.0) is eager
    del t
    gc.collect()
    assert len(hosts) == 1 and hosts[0]() is not None
    # a second graph copies from the same place
    nat._TABLES.clear()
    nat._CONSTANTS.clear()
    gpu.is_in(5, capturing=True)
    make(3.0)
    assert len(hosts) == 1


@pytest.mark.parametrize("make", [constant, plane_table])
def test_table_of_a_captured_graph_outlives_eviction(gpu, make):
    t = make(-1.0)
    addr = weakref.ref(t)
    gpu.is_in(5, capturing=True)
    assert make(-1.0) is t
    assert t.recorded == [] and gpu.log == []
    gpu.is_in(1)
    del t
    for k in range(400):
        make(float(k))
    gc.collect()
    assert addr() is not None
    # a later graph of the same geometry does not displace it
    make(-1.0)
    gpu.is_in(5, capturing=True)
    make(-1.0)
    gpu.is_in(1)
    for k in range(400):
        make(float(k))
    gc.collect()
    assert addr() is not None


@pytest.mark.parametrize("make", [constant, plane_table])
def test_eviction_frees_a_table(gpu, make):
    addr = weakref.ref(make(-1.0))
    for k in range(400):
        make(float(k))
    gc.collect()
    assert addr() is None


def test_constants_do_not_displace_plane_tables(gpu):
    """Many densities or phase factors leave the plane tables where they are."""
    t = plane_table(1.0)
    for k in range(400):
        constant(float(k))
    assert plane_table(1.0) is t
