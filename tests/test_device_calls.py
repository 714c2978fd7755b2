"""What the device-pointer calls of the Python binding hand to the library: only
integers and None are addresses, and every call's options are its own (CPU; the
library call itself is recorded, not made)."""
from __future__ import annotations

import ctypes as C

import numpy as np
import pytest


class Recorder:
    """The library with its device-pointer calls replaced by a note of their options."""

    def __init__(self, lib):
        self.lib, self.seen = lib, []

    def __getattr__(self, name):
        if name not in ("mlem_run_device", "mlem_forward_project", "mlem_back_project"):
            return getattr(self.lib, name)

        def call(*args):
            ro = args[-2]._obj
            self.seen.append({k: getattr(ro, k) for k, _ in ro._fields_})
            return 0

        return call


def unbound(pkg):
    m = object.__new__(pkg.Matrix)
    m._h = C.c_void_p(None)
    return m


@pytest.mark.parametrize("bad", [b"\0" * 64, "text", (C.c_float * 4)(), bytearray(8), np.zeros(4)],
                         ids=["bytes", "str", "array", "bytearray", "ndarray"])
def test_host_memory_is_no_device_pointer(pkg, bad):
    m = unbound(pkg)
    for k in range(3):
        args = [16, 16, 16]
        args[k] = bad
        if k < 2:
            with pytest.raises(TypeError):
                m.run_device(args[0], args[1], 1)
            with pytest.raises(TypeError):
                m.back_project(args[0], args[1])
        with pytest.raises(TypeError):
            m.forward_project(*args)
    with pytest.raises((TypeError, ValueError)):  # an array has no truth value
        m.forward_project(16, 16, 16, bad)
    with pytest.raises((TypeError, ValueError)):
        m.run_device(16, 16, 1, bad)
    m._h = None


def test_options_are_taken_by_value(pkg, monkeypatch):
    torch = pytest.importorskip("torch")
    rec = Recorder(pkg.load_library())
    monkeypatch.setattr(pkg, "load_library", lambda: rec)
    m = unbound(pkg)
    lanes = torch.tensor(8)
    m.run_device(16, 16, 1, lanes=lanes)
    lanes.fill_(16)
    m.run_device(16, 16, 1, lanes=lanes)
    m.back_project(16, 16, lanes=np.array(32))
    m.forward_project(16, 16, 16, kernel=pkg.KERNEL_DIRECT, lanes=4, use_graph=False)
    m.forward_project(16, 16, 16, kernel=pkg.KERNEL_DIRECT, lanes=4, use_graph=0)
    assert [o["lanes"] for o in rec.seen] == [8, 16, 32, 4, 4]
    assert [o["kernel"] for o in rec.seen[3:]] == [pkg.KERNEL_DIRECT] * 2
    m.back_project(16, 16, spmv=0)
    with pytest.raises(TypeError):  # the struct's integer fields take no float, whatever came before
        m.back_project(16, 16, spmv=0.0)
    with pytest.raises(TypeError):
        m.back_project(16, 16, no_such_option=1)
    m._h = None
