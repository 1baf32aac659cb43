"""The bf16 GEMMs over int8 and int4 weights, at the edges of their tiles, against 64-bit torch.

Tolerance: one rounding to bf16 of a sum in f32 (int8; int4 weights are rounded to bf16 first), and a truncated addition per 16 k.
"""

import pytest
import torch

from jax_metallib_b200 import ops

pytestmark = pytest.mark.gpu

# rows at the edges of the tiles (32 to 192) and of their halves; columns of whole and partial channel blocks, few and more
# tiles than SMs; K of one stage, of partial ones and of more than all rings hold
SHAPES = [(33, 64, 24576), (96, 1024, 8192), (161, 1160, 8208), (192, 256, 16384), (193, 640, 8320), (224, 512, 5392),
          (385, 2048, 4096), (777, 384, 6144), (1025, 136, 2064), (1500, 512, 10240)]

# where the kernel for few rows and the GEMM meet, by columns per SM and the length of K
LINE = [(16, 64, 18960), (17, 8, 1024), (17, 64, 976), (20, 72, 4112), (32, 128, 4736), (32, 136, 4752), (31, 520, 9488),
        (33, 1016, 4752), (17, 1032, 14224), (64, 1536, 7120), (17, 2048, 18944), (25, 2056, 18960), (65, 2048, 6336)]

# K split over clusters: few pieces, shares of one stage and of different lengths, edges of rows and columns
SPLIT = [(33, 16384, 128), (40, 8200, 144), (160, 4096, 400), (192, 14336, 1040), (193, 2048, 1792), (300, 1032, 768),
         (500, 5120, 512), (64, 14336, 4096), (1200, 2048, 256)]
# rows in two launches
TWO = [(777, 14336, 4096), (1587, 8192, 5120), (801, 8200, 4112)]


@pytest.mark.parametrize("m,k,n", SHAPES + LINE + SPLIT + TWO)
def test_int8_weights(cuda, m, k, n):
    g = torch.Generator(device="cuda").manual_seed(m + k + n)
    x = torch.randn(m, k, device="cuda", generator=g).bfloat16()
    w = torch.randint(-128, 128, (k, n), dtype=torch.int8, device="cuda", generator=g)
    s = torch.rand(n, device="cuda", generator=g) * 0.01 + 0.005
    wide = torch.full((m, n + 16), 7.0, dtype=torch.bfloat16, device="cuda")
    ops.w8a16_perchannel(x, w, s, out=wide)
    assert bool((wide[:, n:] == 7).all())
    ref, size = (x.double() @ w.double()) * s.double(), (x.double().abs() @ w.double().abs()) * s.double()
    bound = 2.0 ** -8 * ref.abs() + (2 * (k // 16 + 1) + 1) * 2.0 ** -24 * size * 1.01
    assert bool(((wide[:, :n].double() - ref).abs() <= bound).all())


@pytest.mark.parametrize("packed", [True, False])
@pytest.mark.parametrize("m,k,n", [(m, max(128, k // 128 * 128), (n + 127) // 128 * 128) for m, k, n in SHAPES + SPLIT + TWO])
def test_int4_weights(cuda, m, k, n, packed):
    g = torch.Generator(device="cuda").manual_seed(m + k + n)
    x = torch.randn(m, k, device="cuda", generator=g).bfloat16()
    wq = torch.randint(0, 256, (k // 2, n), dtype=torch.uint8, device="cuda", generator=g)
    s = (torch.rand(k // 128, n, device="cuda", generator=g) * 0.008 + 0.002).bfloat16()
    z = torch.randint(0, 16 if packed else 128, (k // 128, n), dtype=torch.uint8, device="cuda", generator=g)
    y = ops.w4a16_g128(x, wq, s, z[:, 0::2] | (z[:, 1::2] << 4) if packed else z, zeros_packed=packed).double()
    q = torch.stack((wq & 15, wq >> 4), 1).reshape(k, n).float()
    # the program's own arithmetic: (q - z) in bf16, exact, times s, rounded to bf16
    w = ((q.bfloat16() - z.repeat_interleave(128, 0).bfloat16()) * s.repeat_interleave(128, 0)).double()
    ref, size = x.double() @ w, x.double().abs() @ w.abs()
    bound = 2.0 ** -8 * ref.abs() + (2 * (k // 16 + 1) + 1) * 2.0 ** -24 * size * 1.01
    assert bool(((y - ref).abs() <= bound).all()), ((y - ref).abs() / bound).max().item()


def test_int8_weights_smallest_activations(cuda):
    """Activations down to the smallest bf16, whose results an ordinary scale brings back."""
    g = torch.Generator(device="cuda").manual_seed(7)
    w = torch.randint(-128, 128, (512, 8192), dtype=torch.int8, device="cuda", generator=g)
    s = (torch.rand(8192, device="cuda", generator=g) + 0.5) * 2.0 ** 100
    for e in (-90, -110, -120, -126, -130, -132):
        x = (torch.randn(130, 512, device="cuda", generator=g).double() * 2.0 ** e).bfloat16()
        y, ref = ops.w8a16_perchannel(x, w, s).double(), (x.double() @ w.double()) * s.double()
        size = (x.double().abs() @ w.double().abs()) * s.double()
        assert bool(((y - ref).abs() <= 2.0 ** -8 * ref.abs() + 70 * 2.0 ** -24 * size).all()), e
