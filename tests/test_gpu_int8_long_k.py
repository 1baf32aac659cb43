"""int8 weights over a long K with few rows: the sums keep the precision that f32 gives.

Which outputs round to another bf16 than the sum in 64 bits: those within the sum's error of the middle between two.  A tensor
core's addition cuts off less than 2^-23 of the sum so far, half of that in the mean, of a sum that is half of the last one in the
mean; the middles are 2^-7.5 of a value apart.  With K / 16 additions in six accumulators that is a share of (K / 96 + 6) * 2^-17.5;
with one accumulator it is more than that (measured: 2.1e-3 for K = 28672, 1.8e-3 for 8192; in six 3e-4 and 3.5e-4).
"""

import pytest
import torch

from jax_metallib_b200 import ops


@pytest.mark.gpu
@pytest.mark.parametrize("m", [17, 24, 32])
@pytest.mark.parametrize("k,n", [(28672, 8192), (8192, 40960)])   # in a cluster; a CTA to a tile
def test_share_of_other_roundings(cuda, m, k, n):
    g = torch.Generator(device="cuda").manual_seed(m)
    x = torch.randn(m, k, device="cuda", generator=g).bfloat16()
    w = torch.randint(-127, 128, (k, n), dtype=torch.int8, device="cuda", generator=g)
    y = ops.w8a16_perchannel(x, w, torch.ones(n, device="cuda"))
    ref = (x.double() @ w.double()).bfloat16()
    assert (y != ref).double().mean().item() < (k / 96 + 6) * 2 ** -17.5


@pytest.mark.gpu
@pytest.mark.parametrize("m,k,n", [(33, 1032, 16384), (64, 1088, 20000), (96, 3000, 18960), (40, 8200, 144), (300, 2056, 4096), (65, 4096, 37904)])
def test_parts(cuda, m, k, n):
    """Tiles of 32 to 96 rows, K of one stage more than a part, of parts of different lengths, in slices and whole; several tiles to a CTA."""
    g = torch.Generator(device="cuda").manual_seed(m + k)
    x = torch.randn(m, k, device="cuda", generator=g).bfloat16()
    w = torch.randint(-128, 128, (k, n), dtype=torch.int8, device="cuda", generator=g)
    s = torch.rand(n, device="cuda", generator=g) * 0.01 + 0.005
    y = ops.w8a16_perchannel(x, w, s).double()
    ref, size = (x.double() @ w.double()) * s.double(), (x.double().abs() @ w.double().abs()) * s.double()
    bound = 2.0 ** -8 * ref.abs() + (2 * (k // 16 + 1) + 1) * 2.0 ** -24 * size * 1.01
    assert bool(((y - ref).abs() <= bound).all())
