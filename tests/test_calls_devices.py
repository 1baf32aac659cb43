"""Devices of the operands of ``ops`` and ``quantized``: no kernel is pointed at another device's memory."""

import re
from pathlib import Path

import pytest
import torch

from jax_metallib_b200 import _calls, ops

SOURCE = (Path(__file__).parent.parent / "jax_metallib_b200" / "binding" / "calls.cc").read_text()


def test_one_device():
    def cuda(*numbers):
        return [torch.device("cuda", n) for n in numbers]

    assert _calls.one_device(1, *cuda(1, 1, 1))
    assert not _calls.one_device(1, *cuda(1, 0, 1))      # weights elsewhere
    assert not _calls.one_device(1, *cuda(1, 1, 1, 2))   # biases elsewhere
    assert not _calls.one_device(0, *cuda(1, 1, 1))      # not the current device
    assert not _calls.one_device(0, *cuda(0, 0), torch.device("cpu"))
    with pytest.raises(TypeError):
        _calls.one_device(0, 1)


def test_every_call_asks():
    """No compiled call looks at a tensor argument but through the function that compares devices."""
    calls = re.findall(r"^PyObject\* (\w+)\(PyObject\*, PyObject\* const\* a, Py_ssize_t n\) \{(.*?)^\}", SOURCE, re.M | re.S)
    assert len(calls) >= 8
    for name, body in calls:
        if name not in ("bind", "one_device"):
            assert "operands(a, " in body and "plain(a[" not in body, name


class _On(torch.Tensor):
    """A host tensor that says it is on a CUDA device."""

    is_cuda = True
    device = property(lambda self: torch.device("cuda", self.number))


def test_mixed_devices_are_refused():
    def on(number, t):
        t = t.as_subclass(_On)
        t.number = number
        return t

    x, w, s = on(0, torch.ones(4, 16)), on(0, torch.ones(16, 16, dtype=torch.int8)), on(1, torch.ones(16))
    ops._need_cuda(x, w, None)
    with pytest.raises(ValueError, match="on one device"):
        ops.w8a32_perchannel(x, w, s)
    with pytest.raises(ValueError, match="on one device"):
        ops.i8_dot(w, on(1, torch.ones(16, 16, dtype=torch.int8)))
