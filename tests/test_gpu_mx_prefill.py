"""The MX matmul that converts its weights into tensor memory, at the edges of its tiles, rings, units and slices, against
64-bit torch.

Tolerance: products are exact; an accumulator takes 32 truncated additions in a unit of 512 k, units and up to eight slices are
added in f32, and the result is rounded to f16 once.
"""

import pytest
import torch

from jax_metallib_b200 import quantized

pytestmark = pytest.mark.gpu

BITS = {"mxfp4": 4, "mxfp8": 8, "nvfp4": 4}


def _weights(mode, n, k, g, lo=110, hi=120):
    """Packed weights, scales and the weights [N, K] in 64 bits."""
    if mode == "mxfp8":
        packed = (torch.randn(n, k, device="cuda", generator=g) * 100).clamp(-448, 448).to(torch.float8_e4m3fn).view(torch.uint8)
        values = packed.view(torch.float8_e4m3fn).double()
    else:
        codes = torch.randint(0, 16, (n, k), dtype=torch.uint8, device="cuda", generator=g)
        packed = codes[:, 0::2] | (codes[:, 1::2] << 4)
        table = torch.tensor([0, .5, 1, 1.5, 2, 3, 4, 6], device="cuda", dtype=torch.float64)
        values = torch.cat((table, -table))[codes.long()]
    if mode == "nvfp4":
        scales = torch.randint(8, 64, (n, k // 16), dtype=torch.uint8, device="cuda", generator=g)
        return packed, scales, values * scales.view(torch.float8_e4m3fn).double().repeat_interleave(16, 1)
    scales = torch.randint(lo, hi, (n, k // 32), dtype=torch.uint8, device="cuda", generator=g)
    return packed, scales, values * torch.exp2(scales.double() - 127).repeat_interleave(32, 1)


def _check(mode, x, packed, scales, w):
    y = quantized.quantized_matmul(x, packed, scales, mode=mode, K=x.shape[1]).double()
    ref, size = x.double() @ w.T, x.double().abs() @ w.abs().T
    bound = 2.0 ** -11 * ref.abs() + 2.0 ** -24 + (2 * 32 + x.shape[1] / 512 + 8) * 2.0 ** -24 * size
    assert bool(((y - ref).abs() <= bound).all()), ((y - ref).abs() / bound).max().item()


# rows at the edges of the tiles (16 to 192) and of their halves; K of one unit, of several and of parts of one, odd numbers of
# 32; columns ragged, odd, in one tile, in more tiles than SMs; K in one slice and in several
@pytest.mark.parametrize("m,k,n", [(5, 32, 128), (16, 512, 96), (17, 96, 130), (33, 1056, 1), (64, 4096, 257), (65, 544, 640),
                                   (129, 2080, 200), (176, 1536, 9600), (193, 160, 19200), (300, 14336, 128), (385, 608, 6401),
                                   (577, 1024, 384)])
@pytest.mark.parametrize("mode", sorted(BITS))
def test_edges(cuda, mode, m, k, n):
    g = torch.Generator(device="cuda").manual_seed(m + k + n)
    x = torch.randn(m, k, device="cuda", generator=g).half()
    _check(mode, x, *_weights(mode, n, k, g))


@pytest.mark.parametrize("m,k,n", [(24, 2048, 160), (150, 1024, 19200)])   # K in slices; one CTA to a tile
@pytest.mark.parametrize("mode", ["mxfp4", "mxfp8"])
def test_scales_far_apart(cuda, mode, m, k, n):
    """A group of zeros with a scale far above its neighbours': what f16 cannot hold beside it is not lost.  These columns are
    computed with k additions in a row; groups within the range (20 powers of two here) are not."""
    g = torch.Generator(device="cuda").manual_seed(m)
    packed, scales, w = _weights(mode, n, k, g, 100, 121)
    per_group = 32 * BITS[mode] // 8
    far = torch.arange(0, n, 37, device="cuda")
    for group in (3, 20):
        packed[far, group * per_group:(group + 1) * per_group] = 0
        scales[far, group] = 200
        w[far, 32 * group:32 * (group + 1)] = 0
    scales[1], w[1] = 0, w[1] * torch.exp2(-scales[1].double()).repeat_interleave(32, 0)   # all groups at 2^-127
    x = (torch.randn(m, k, device="cuda", generator=g) * 8).half()
    y = quantized.quantized_matmul(x, packed, scales, mode=mode, K=k).double()
    ref, size = x.double() @ w.T, x.double().abs() @ w.abs().T
    bound = 2.0 ** -11 * ref.abs() + 2.0 ** -24 + (k + 8) * 2.0 ** -24 * size
    assert bool(((y - ref).abs() <= bound).all()), ((y - ref).abs() / bound).max().item()
    assert bool((y[:, far].abs().amax(0) > 2.0 ** -10).all())
