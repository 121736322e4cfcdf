"""`refresh_device`'s host copy of the coefficients, on the CPU: torch and the
library are stood in for by a stream that runs its work only when it is waited
for, so a copy that nobody waits for never arrives.

On a stream of torch's that has a handle the library runs, and waits for, that
stream; on torch's default stream (handle 0) it runs on its own, and its call
completes nothing that is queued on the default stream."""
import types

import numpy as np
import pytest

from tpagmg import projection as P


class Stream:
    def __init__(self, handle):
        self.cuda_stream, self.work = handle, []

    def synchronize(self):
        while self.work:
            self.work.pop(0)()


class Tensor:
    """float64 device or pinned array; copies run on `stream`."""

    def __init__(self, data, stream):
        self.data, self.stream = data, stream
        self.shape, self.dtype, self.device = data.shape, data.dtype, "cuda:0"

    def detach(self):
        return self

    def data_ptr(self):
        return self.data.ctypes.data

    def numpy(self):
        return self.data

    def copy_(self, src, non_blocking=False):
        self.stream.work.append(lambda: self.data.__setitem__(..., src.data))
        if not non_blocking:
            self.stream.synchronize()
        return self

    def cpu(self):
        out = Tensor(np.zeros(self.shape), self.stream)
        return out.copy_(self)


def setup(handle, monkeypatch, fails=False):
    stream = Stream(handle)
    torch = types.SimpleNamespace(
        cuda=types.SimpleNamespace(current_stream=lambda device=None: stream),
        empty=lambda shape, dtype=None, pin_memory=False, **kw: Tensor(np.zeros(shape), stream))
    monkeypatch.setattr(P, "_torch", lambda: torch)

    def call(name, *args):
        if handle:  # the library runs on torch's stream and waits for it
            stream.synchronize()
        if fails:
            raise RuntimeError(name)

    solver = types.SimpleNamespace(device=0, set_stream=lambda h: None, ctx=types.SimpleNamespace(call=call),
                                   operator=types.SimpleNamespace(face_coefficient=np.full(5, -1.0)))
    return stream, solver, Tensor(np.arange(5.0), stream)


@pytest.mark.parametrize("handle", [0, 0x1234])
def test_coefficients_have_arrived(handle, monkeypatch):
    stream, solver, kappa = setup(handle, monkeypatch)
    P.refresh_device(solver, kappa)
    assert not stream.work  # the next kernel that writes kappa finds no copy reading it
    assert np.array_equal(solver.operator.face_coefficient, np.arange(5.0))
    kappa.data[:] = 7.0
    assert np.array_equal(solver.operator.face_coefficient, np.arange(5.0))


def test_a_failed_refresh_keeps_the_coefficients(monkeypatch):
    stream, solver, kappa = setup(0, monkeypatch, fails=True)
    with pytest.raises(RuntimeError):
        P.refresh_device(solver, kappa)
    assert not stream.work
    assert np.array_equal(solver.operator.face_coefficient, np.full(5, -1.0))
