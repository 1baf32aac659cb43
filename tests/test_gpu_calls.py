"""The compiled calls of ops.py and quantized.py against the Python code that takes what they decline."""

import pytest
import torch

from jax_metallib_b200 import _calls, ops, quantized

pytestmark = pytest.mark.gpu


def _calls_of(m, k, n, g):
    """Name -> (function of the activations, activations)."""
    def rand(*shape, dtype=torch.float32):
        return torch.randn(*shape, device="cuda", generator=g).to(dtype)

    def byte(*shape, dtype=torch.uint8, hi=255):
        return torch.randint(0, hi, shape, device="cuda", generator=g, dtype=torch.uint8).view(dtype)

    w, s, row = byte(k, n, dtype=torch.int8), rand(n).abs(), rand(m).abs()
    wq, s4, z4 = byte(k // 2, n), rand(k // 128, n, dtype=torch.bfloat16), byte(k // 128, n // 2)
    p4, p8 = byte(n, k // 8 * 4).view(torch.int32), byte(n, k)
    sc, bi = rand(n, k // 64), rand(n, k // 64)
    e8 = torch.randint(118, 125, (n, k // 32), dtype=torch.uint8, device="cuda", generator=g)
    return {
        "w8a32": (lambda x: ops.w8a32_perchannel(x, w, s), rand(m, k)),
        "w8a16": (lambda x: ops.w8a16_perchannel(x, w, s), rand(m, k, dtype=torch.bfloat16)),
        "i8_acc": (lambda x: ops.i8_dot(x, w)[0], byte(m, k, dtype=torch.int8)),
        "i8_unsigned": (lambda x: ops.i8_dot(x, w, row, s, want_acc=False)[1], byte(m, k)),
        "w4a16": (lambda x: ops.w4a16_g128(x, wq, s4, z4, zeros_packed=True, static_weights=True), rand(m, k, dtype=torch.bfloat16)),
        "affine4": (lambda x: quantized.affine_quantized_matmul(x, p4, sc, bi, bits=4, group_size=64, K=k), rand(m, k, dtype=torch.float16)),
        "affine8": (lambda x: quantized.affine_quantized_matmul(x, p8, sc, bi, bits=8, group_size=64, K=k), rand(m, k)),
        "mxfp8": (lambda x: quantized.quantized_matmul(x, p8 & 0x77, e8, mode="mxfp8", K=k), rand(m, k, dtype=torch.float16)),
        "mxfp4": (lambda x: quantized.quantized_matmul(x, wq.view(-1)[:n * k // 2].view(n, k // 2), e8, mode="mxfp4", K=k), rand(m, k)),
    }


class _Declines:
    def __getattr__(self, name):
        return lambda *args: None


@pytest.mark.parametrize("m", [1, 5, 40])
@pytest.mark.parametrize("n", [512, 24576])   # int4 without and with a workspace
def test_same_results(cuda, monkeypatch, m, n):
    g = torch.Generator(device="cuda").manual_seed(m)
    for name, (call, x) in _calls_of(m, 512, n, g).items():
        y = call(x)
        with monkeypatch.context() as mp:
            mp.setattr(ops, "_calls", _Declines())
            for compiled in ("mx_matmul", "affine_matmul"):
                mp.setattr(_calls, compiled, lambda *args: None)
            z = call(x)
        assert y.shape == z.shape and y.dtype == z.dtype and y.is_contiguous() and torch.equal(y, z), name
        offset = torch.cat((x.view(-1)[:512], x.view(-1)))[512:].view(x.shape)   # storage that does not begin with the tensor
        assert torch.equal(call(offset), y), name
        assert torch.equal(call(torch.nn.Parameter(x, requires_grad=False)), y), name


def test_leading_dimensions(cuda):
    g = torch.Generator(device="cuda").manual_seed(2)
    calls = _calls_of(6, 512, 256, g)
    for name in ("w8a32", "affine4", "affine8", "mxfp8"):
        call, x = calls[name]
        assert torch.equal(call(x.view(2, 3, 512)), call(x).view(2, 3, 256))
        assert call(x[0]).shape == (256,)


def test_declined(cuda):
    """What is not a plain tensor goes the way it went, errors and all."""
    g = torch.Generator(device="cuda").manual_seed(3)
    w, s = torch.ones(64, 32, dtype=torch.int8, device="cuda"), torch.ones(32, device="cuda")
    x = torch.randn(4, 64, device="cuda", generator=g)
    with pytest.raises(ValueError, match="contiguous"):
        ops.w8a32_perchannel(x.t().contiguous().t(), w, s)
    with pytest.raises(TypeError, match="expected x float32"):
        ops.w8a32_perchannel(x.half(), w, s)
    with pytest.raises(ValueError, match="shape mismatch"):
        ops.w8a32_perchannel(x[:, :32].contiguous(), w, s)
    with pytest.raises(TypeError, match="CUDA tensors only"):
        ops.w8a32_perchannel(x.cpu(), w, s)
    with pytest.raises(ValueError, match="go together"):
        ops.i8_dot(w, w.t().contiguous(), s, None)
    assert ops.w8a32_perchannel(x[:0], w, s).shape == (0, 32)

    class Sub(torch.Tensor):
        pass

    assert _calls.w8a32(x.as_subclass(Sub), w, s) is None
    seen = []

    class Mode(torch.utils._python_dispatch.TorchDispatchMode):
        def __torch_dispatch__(self, func, types, args=(), kwargs=None):
            seen.append(func)
            return func(*args, **(kwargs or {}))

    with Mode():
        assert _calls.w8a32(x, w, s) is None
        y = ops.w8a32_perchannel(x, w, s)
    assert any("empty" in str(f) for f in seen) and torch.equal(y, ops.w8a32_perchannel(x, w, s))
    with pytest.raises(RuntimeError):
        torch.vmap(lambda row: ops.w8a32_perchannel(row[None], w, s))(x)
