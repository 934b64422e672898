"""CPU: the bench reads an event pair only when the later event is known to be
complete.  The library may have finished on a stream of its own before the event
recorded behind the call on the caller's stream has, so waiting for the library
is not enough."""
import types

import numpy as np

import bench


class _Event:
    def __init__(self, enable_timing=False):
        self.done = False

    def record(self, stream=None):
        self.done = False

    def synchronize(self):
        self.done = True

    def elapsed_time(self, other):
        if not other.done:
            raise RuntimeError("Both events must be completed before calculating elapsed time.")
        return 1.0


class _Buffer:
    def __init__(self, size):
        self.size = size

    def zero_(self):
        pass

    def data_ptr(self):
        return 0

    def cpu(self):
        return self

    def numpy(self):
        return np.zeros(self.size, np.uint8)

    def __getitem__(self, _):
        return self


def _torch():
    torch = types.SimpleNamespace(uint8=None, empty=lambda n, **kw: _Buffer(n))
    torch.cuda = types.SimpleNamespace(Event=_Event, synchronize=lambda: None)
    return torch


class _Ctx:
    ptr = lib = None
    sync = staticmethod(lambda: None)
    last_kernel_ms = staticmethod(lambda: 1.0)
    last_stage_ms = staticmethod(lambda: [0.0] * 3)
    last_passes_ms = staticmethod(lambda: [0.0] * 4)


def test_timer_waits_for_its_own_event():
    timer = bench.Timer(_torch(), None, _Ctx(), 1, None)
    step_ms, kern_ms, _ = timer.run(3, lambda: None)
    assert step_ms == [1.0] * 3 and kern_ms == [1.0] * 3


def test_graph_replay_waits_for_its_own_event(monkeypatch):
    import sdim_gb300.graph as graph

    class _Run:
        def __init__(self, *a, **kw):
            pass

        launch = staticmethod(lambda **kw: None)
        sync = close = staticmethod(lambda: None)
        info = staticmethod(lambda: {"nodes": 1, "kernel_nodes": 1})

    monkeypatch.setattr(graph, "CapturedRun", _Run)
    torch = _torch()
    timer = bench.Timer(torch, None, _Ctx(), 1, None)
    entry = types.SimpleNamespace(shots=4, shot0=0, program=types.SimpleNamespace(num_records=2))
    out = bench.graph_replay(types.SimpleNamespace(steps=2, warmup=1), torch, _Ctx(), timer,
                             types.SimpleNamespace(cuda_stream=0), [entry], 1, lambda: np.zeros(9, np.uint8))
    assert out["ms_per_step"] == 1.0
