"""The device entry points take objects with data_ptr() and nothing else: the address of
a host array must not reach a kernel. Runs against a stub of the library."""
import ctypes

import numpy as np
import pytest

import xrt_rs
from xrt_rs import _lib


class Ctx:
    handle = None


class Tensor:
    """Stands for a device tensor."""

    def __init__(self, at):
        self.at = at

    def data_ptr(self):
        return self.at

    def numel(self):
        return 4


@pytest.fixture
def calls(monkeypatch):
    got = []

    class Lib:
        def xk_diffraction_integral_device(self, handle, rays, n, pix, m, out, path, stream, st):
            got.append([ctypes.cast(f._obj.__getattribute__(name), ctypes.c_void_p).value
                        for f in (rays, pix, out) for name, _ in f._obj._fields_])
            return 0

    monkeypatch.setattr(_lib, "load", lambda: Lib())
    monkeypatch.setattr(_lib, "check", lambda rc, handle=None: None)
    return got


def columns(kind):
    if kind == "tensors":
        return [[Tensor(64 * (10 * a + i + 1)) for i in range(n)]
                for a, n in enumerate((12, 3, 4))]
    return [[np.zeros(4) for _ in range(n)] for n in (12, 3, 4)]


@pytest.mark.parametrize("host", [0, 1, 2])
def test_host_arrays_are_refused(calls, host):
    args = columns("tensors")
    args[host][-1] = columns("arrays")[host][-1]
    with pytest.raises(AttributeError):
        xrt_rs.diffraction_integral_device(*args, ctx=Ctx())
    with pytest.raises(AttributeError):
        xrt_rs.diffraction_integral_device(*columns("arrays"), ctx=Ctx())
    assert calls == []


def test_tensors_arrive_in_order(calls):
    args = columns("tensors")
    xrt_rs.diffraction_integral_device(*args, ctx=Ctx())
    assert calls == [[t.at for group in args for t in group]]


def test_missing_columns_are_null_and_surplus_ones_an_error(calls):
    args = columns("tensors")
    args[0].pop()
    xrt_rs.diffraction_integral_device(*args, ctx=Ctx())  # the library refuses the null
    assert calls[0][11] is None
    args[0] += [Tensor(1), Tensor(2)]
    with pytest.raises(TypeError):
        xrt_rs.diffraction_integral_device(*args, ctx=Ctx())
    assert len(calls) == 1
