"""The compiled calls are a convenience: the library is built, and the operators work, without them."""

import os
import subprocess
import sys
import types

import pytest

from jax_metallib_b200 import _lib, build

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def _python(code):
    return subprocess.run([sys.executable, "-W", "default", "-c", code], cwd=ROOT, capture_output=True, text=True)


def test_library_is_built_without_torch(monkeypatch, tmp_path):
    monkeypatch.setitem(sys.modules, "torch", None)   # import torch raises ImportError
    for name in ("CALLS", "CALLS_KEY"):
        monkeypatch.setattr(build, name, str(tmp_path / name))
        (tmp_path / name).write_text("of another torch")
    assert build.build() == build.LIB and os.path.exists(build.LIB)
    assert not os.path.exists(build.CALLS)
    cpu_only = types.ModuleType("torch")
    cpu_only.version = types.SimpleNamespace(cuda=None)
    monkeypatch.setitem(sys.modules, "torch", cpu_only)
    assert build.build_calls() is None


def test_key_names_what_a_binary_depends_on():
    keys = {build.calls_key(*of) for of in (("2.11.0", "12.8", 1), ("2.12.0", "12.8", 1), ("2.11.0", "13.0", 1), ("2.11.0", "12.8", 0))}
    assert len(keys) == 4
    torch = pytest.importorskip("torch")
    build.build_calls()
    assert open(build.CALLS_KEY).read() == build.calls_key(torch.__version__, torch.version.cuda, int(torch._C._GLIBCXX_USE_CXX11_ABI))


@pytest.mark.parametrize("spoil", ["sys.modules['jax_metallib_b200._calls'] = None",                          # no such file
                                   "from jax_metallib_b200 import _calls; _calls.TORCH = '1.0'"])   # built for another torch
def test_operators_import_without_it(spoil):
    done = _python(f"""
import sys, torch
{spoil}
from jax_metallib_b200 import _lib, ops, quantized
assert ops._calls.w8a32(1, 2, 3) is None
_lib.bind_calls()
try:
    ops.w8a32_perchannel(torch.ones(1, 1), torch.ones(1, 1), torch.ones(1))
except TypeError as e:
    print(e)
""")
    assert done.returncode == 0, done.stderr
    assert "CUDA tensors only" in done.stdout and "_calls.so is not used" in done.stderr


def test_it_is_used_here():
    pytest.importorskip("torch")
    assert not isinstance(_lib.calls(), _lib._Declines)
