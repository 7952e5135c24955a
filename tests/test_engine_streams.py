"""How the engine orders its streams, against a fake of the native calls (no GPU)."""
from types import SimpleNamespace

import pytest
import torch

import hipress_b200 as hp
from hipress_b200._native.lib import NativeLibraryError
from hipress_b200.config import HipressConfig
from hipress_b200.parallel import engine as engine_module
from hipress_b200.parallel.engine import GradSyncEngine

HERE, COMM = 11, 22     # stream handles


class Native:
    def __init__(self, rc=0):
        self.rc, self.calls = rc, []

    def stream_order(self, event, src, dst):
        self.calls.append(("order", src, dst))
        return self.rc


def _engine(monkeypatch, native):
    """An engine of CPU parameters dressed up as one with a fused bucket on a GPU."""
    hp.init()
    monkeypatch.setattr(engine_module, "stream_ptr", lambda stream=None: HERE)
    named = [("w", torch.nn.Parameter(torch.zeros(300))), ("b", torch.nn.Parameter(torch.zeros(20)))]
    eng = GradSyncEngine(named, HipressConfig(algorithm="tbq", comp_threshold=1, overlap=False))
    eng._fast, eng._order = native, [SimpleNamespace(handle=100 + i) for i in range(len(eng.buckets) + 1)]
    eng.comm_stream = SimpleNamespace(cuda_stream=COMM)
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
