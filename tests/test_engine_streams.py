"""How the engine orders its streams, against a fake of the native calls (no GPU)."""
from types import SimpleNamespace

import pytest
import torch

import hipress_b200 as hp
from hipress_b200._native import lib
from hipress_b200._native.lib import NativeLibraryError
from hipress_b200.config import HipressConfig
from hipress_b200.parallel import engine as engine_module
from hipress_b200.parallel.engine import GradSyncEngine

HERE, COMM = 11, 22     # stream handles


class Event(dict):
    """Stands for an OrderEvent: its handle names the device it was made on."""

    def __missing__(self, device):
        return 1000 + device


class Native:
    def __init__(self, rc=0):
        self.rc, self.calls, self.events = rc, [], []

    def stream_order(self, event, src, dst):
        self.calls.append(("order", src, dst))
        self.events.append(event)
        return self.rc


def _engine(monkeypatch, native):
    """An engine of CPU parameters dressed up as one with a fused bucket on a GPU."""
    hp.init()
    monkeypatch.setattr(engine_module, "stream_ptr", lambda stream=None: HERE)
    monkeypatch.setattr(engine_module, "current_device", lambda: 1, raising=False)
    named = [("w", torch.nn.Parameter(torch.zeros(300))), ("b", torch.nn.Parameter(torch.zeros(20)))]
    eng = GradSyncEngine(named, HipressConfig(algorithm="tbq", comp_threshold=1, overlap=False))
    eng._fast, eng._order = native, [Event() for _ in range(len(eng.buckets) + 1)]
    eng.comm_stream = SimpleNamespace(cuda_stream=COMM, device_index=3)
    eng.on_cuda = True
    for b in eng.buckets:
        b.impl = SimpleNamespace(launch_ptrs=lambda *a, **k: native.calls.append(("launch",)))
        eng.make_launch_args(b)
    for _, p in named:
        p.grad = torch.ones_like(p)
    return eng


def test_a_failed_ordering_in_front_of_a_launch_raises(monkeypatch):
    native = Native(rc=400)     # cudaErrorInvalidResourceHandle
    eng = _engine(monkeypatch, native)
    with pytest.raises(NativeLibraryError, match="stream order"):
        eng.synchronize()
    assert native.calls == [("order", HERE, COMM)], "nothing is launched that is not ordered"


def test_a_failed_ordering_behind_the_launches_raises(monkeypatch):
    native = Native()
    eng = _engine(monkeypatch, native)
    launch = eng._launch

    def last_one_fails(b):
        launch(b)
        native.rc = 400
    eng._launch = last_one_fails
    with pytest.raises(NativeLibraryError, match="stream order"):
        eng.synchronize()
    assert native.calls[-1] == ("order", COMM, HERE)


def test_events_belong_to_the_device_of_the_stream_they_record(monkeypatch):
    """The device that is current at a step may be another than the communication
    stream's, and than the one that was current when the engine was built."""
    native = Native()
    _engine(monkeypatch, native).synchronize()
    assert native.calls == [("order", HERE, COMM), ("launch",), ("order", COMM, HERE)]
    assert native.events == [1001, 1003]


def test_an_order_event_is_made_once_on_each_device(monkeypatch):
    made, current = [], [0]

    class Device:
        def __init__(self, d):
            self.d = d

        def __enter__(self):
            self.before, current[0] = current[0], self.d

        def __exit__(self, *a):
            current[0] = self.before

    def create(out):
        made.append(current[0])
        out._obj.value = 500 + current[0]
        return 0
    native = SimpleNamespace(hp_cuda_event_create=create, hp_cuda_event_destroy=lambda h: made.append(-h))
    monkeypatch.setattr(torch.cuda, "device", Device)
    monkeypatch.setattr(lib, "current_device", lambda: current[0], raising=False)
    monkeypatch.setattr(lib, "cuda", lambda: native)
    monkeypatch.setattr(lib, "_cuda", native)
    e = lib.OrderEvent()
    assert [e[0], e[2], e[2], e[0]] == [500, 502, 502, 500] and made == [0, 2]
    del e
    assert sorted(made[2:]) == [-502, -500]


def test_missing_gradients_are_made_before_the_ordering(monkeypatch):
    """A gradient that does not exist yet is filled on the caller's stream; the kernel on
    the communication stream must run behind that fill."""
    native = Native()
    eng = _engine(monkeypatch, native)
    grad = eng._grad

    def recorded(e):
        native.calls.append(("grad", e.name))
        return grad(e)
    eng._grad = recorded
    for e in eng.entries:
        e.param.grad = None
    eng.synchronize()
    kinds = [c[0] for c in native.calls]
    assert kinds == ["grad"] * len(eng.entries) + ["order", "launch", "order"]
    assert all(e.param.grad is not None for e in eng.entries)


def test_flat_syncer_fills_new_state_on_the_kernels_stream(monkeypatch):
    """The caller orders `stream` behind the gradient, not behind state that the first call
    makes: that has to be filled on the same stream."""
    import contextlib
    from hipress_b200.parallel import hooks
    current, made = [None], []

    @contextlib.contextmanager
    def on(stream):
        before, current[0] = current[0], stream
        yield
        current[0] = before
    hp.init()
    monkeypatch.setattr(torch.cuda, "stream", on)
    for name in ("zeros", "empty"):
        def recorded(*a, _make=getattr(torch, name), **k):
            made.append(current[0])
            return _make(*a, **k)
        monkeypatch.setattr(hooks.torch, name, recorded)
    fs = hooks.FlatSyncer(HipressConfig(algorithm="dgc", topology="ps", comp_threshold=0, server_residual=False))
    launched = []
    impl = SimpleNamespace(sizes=[5000], launch_ptrs=lambda *a, **k: launched.append(k["stream"]))

    def fused_impl(key, n, device):
        if key not in fs._fused:
            made.append(current[0])
        return fs._fused.setdefault(key, (impl, None, None))
    fs._fused_impl = fused_impl
    flat = torch.ones(5000)
    for _ in range(2):
        fs._sync_fused(flat, 0, COMM)
    # momentum, accumulator, kernel scratch, the owner's accumulator: once each
    assert launched == [COMM, COMM] and made == [COMM] * 4


def test_an_encode_on_another_stream_makes_its_workspace_there(monkeypatch):
    import contextlib
    from hipress_b200.ops import compressor
    current, made = [None], []

    @contextlib.contextmanager
    def on(stream):
        before, current[0] = current[0], stream
        yield
        current[0] = before
    monkeypatch.setattr(torch.cuda, "stream", on)
    monkeypatch.setattr(compressor._lib, "fast_cuda", lambda: SimpleNamespace(sparse_encode=lambda *a: 0))
    monkeypatch.setattr(compressor._lib, "stream_ptr", lambda stream=None: HERE)
    c = compressor.Compressor("graddrop", ratio=0.1)
    c.new_workspace = lambda device, n=None: made.append(current[0]) or torch.zeros(8, dtype=torch.int32)
    g = SimpleNamespace(numel=lambda: 100, is_cuda=True, device="cuda", data_ptr=lambda: 0)
    state = {"residual": torch.zeros(100)}
    for stream in (None, COMM):
        c._encode_sparse(g, state, None, torch.zeros(200, dtype=torch.uint8), True, None, None, stream, 0)
    assert made == [None, COMM]
