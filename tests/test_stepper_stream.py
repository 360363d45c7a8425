"""A stepper on a stream of its own: what its constructor fills (the clock, the work arrays) is
filled on that stream, after what the caller had in flight and ahead of the first kernel; a
clock made by itself is complete when its constructor returns.  The order of the calls is
recorded without a device; on one, such a stepper gives the bits of one on the current stream."""
import contextlib
import ctypes
import types

import numpy as np
import pytest
import torch

import phd_code_gb300 as pkg
from _util import lattice_mesh, smooth_state
from phd_code_gb300 import _lib as L
from phd_code_gb300 import device, step


class Recorder:
    """Stands in for the streams and the library: who launched or filled what, and where."""

    def __init__(self, monkeypatch):
        self.log, self.current = [], "default"
        rec = self

        class Lib:
            def __getattr__(self, name):
                def call(*a):
                    rec.log.append((name, rec.current if not rec.handles else rec.handles.pop()))
                    return 0
                return call

        def stream_handle(stream=None, device=None):
            self.handles.append(self.current if stream is None else stream.name)
            return ctypes.c_void_p(0)

        @contextlib.contextmanager
        def on(stream):
            before, self.current = self.current, stream.name if stream is not None else self.current
            yield
            self.current = before

        self.handles = []
        monkeypatch.setattr(L, "lib", lambda: Lib())
        monkeypatch.setattr(L, "stream_handle", stream_handle)
        for mod in (device, step):
            monkeypatch.setattr(mod, "_dev", lambda d: torch.device("cpu"), raising=False)
        monkeypatch.setattr(torch.cuda, "stream", on)
        monkeypatch.setattr(torch.cuda, "current_stream", lambda d=None: self.stream(self.current))
        zeros, fill, copy = torch.zeros, torch.Tensor.fill_, torch.Tensor.copy_

        def logged(name, f):
            def call(*a, **k):
                self.log.append((name, self.current))
                return f(*a, **k)
            return call

        monkeypatch.setattr(torch, "zeros", logged("zeros", zeros))
        monkeypatch.setattr(torch.Tensor, "fill_", logged("fill", fill))
        monkeypatch.setattr(torch.Tensor, "copy_", logged("host copy", copy))

    def stream(self, name):
        return types.SimpleNamespace(name=name, cuda_stream=0,
                                     wait_stream=lambda other: self.log.append(("wait for " + other.name, name)),
                                     wait_event=lambda e: None, synchronize=lambda: None)


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
def test_constructor_fills_on_the_steppers_stream(precision, monkeypatch):
    mesh = lattice_mesh(6, "periodic", seed=1)
    rec = Recorder(monkeypatch)
    st = pkg.FluxStepper(mesh, smooth_state(mesh), precision=precision, device="cpu", stream=rec.stream("own"))
    assert st.stream.name == "own"
    names = [n for n, _ in rec.log]
    assert "wait for default" in names and "zeros" in names and "phd_cons_from_prim_f64" in names
    after = rec.log[names.index("wait for default"):]
    assert [x for x in rec.log if x[0].startswith(("zeros", "fill", "phd_"))] == \
        [x for x in after if x[0].startswith(("zeros", "fill", "phd_"))]
    assert all(where == "own" for n, where in after)
    del rec.log[:]
    pkg.FluxStepper(mesh, smooth_state(mesh), precision=precision, device="cpu")
    assert all(where == "default" and not n.startswith("wait") for n, where in rec.log)


def test_a_clock_by_itself_is_complete(monkeypatch):
    rec = Recorder(monkeypatch)
    device.DeviceClock("cpu")
    assert rec.log[-1][0] == "host copy"                  # pageable memory: the call returns after it
    c = device.DeviceClock("cpu", dt=0.5, t=1.0, t_end=2.0).read()
    assert (c.dt, c.t, c.t_end, c.status, c.step, c.arrive) == (0.5, 1.0, 2.0, 0, 0, 0)
    for k in (dict(), dict(in_stream=True)):
        c = device.DeviceClock("cpu", **k).read()
        assert (c.dt, c.t, c.t_end, c.dt_last, c.status, c.step, c.arrive) == (0.0,) * 4 + (0,) * 3
        assert c.dtmin_bits == np.float64(np.inf).view(np.uint64)


@pytest.mark.gpu
@pytest.mark.parametrize("precision", ["fp64", "fp32"])
def test_own_stream_equals_the_current_one(precision):
    mesh = lattice_mesh(40, "periodic", seed=1)
    prim = smooth_state(mesh)
    a = pkg.FluxStepper(mesh, prim, precision=precision, moving=True)
    a.step(3)
    own = torch.cuda.Stream()
    busy = torch.zeros(1 << 26, device="cuda")
    dm = pkg.DeviceMesh(mesh)
    for _ in range(50):
        busy.add_(1.0)                                    # work in flight on the current stream
    b = pkg.FluxStepper(dm, prim, precision=precision, moving=True, stream=own)
    b.step(3)
    own.synchronize()
    assert np.array_equal(a.cons_host(), b.cons_host()) and a.read_clock().dt == b.read_clock().dt
