"""int4 weights with 9 to 32 rows: two tiles of 16 rows side by side, and the lines between the kernels, against 64-bit torch.

Tolerance: one rounding to bf16 of a sum in f32, whose products are x (q - z) or, in the kernel for wide matrices, x q and x z.
"""

import pytest
import torch

from jax_metallib_b200 import ops

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("packed", [True, False])
@pytest.mark.parametrize("m,k,n", [(17, 128, 512), (24, 256, 256), (25, 1024, 1024), (31, 4096, 384), (32, 4096, 10240),
                                   (32, 4096, 10368), (29, 2048, 12416), (18, 2176, 12416), (32, 14336, 2048), (17, 512, 38016),
                                   (9, 1024, 18944), (13, 1024, 19072), (16, 28672, 2816), (8, 28672, 2816)])
def test_rows(cuda, m, k, n, packed):
    g = torch.Generator(device="cuda").manual_seed(m + k + n)
    x = (torch.randn(m, k, device="cuda", generator=g) * 3 + 1).bfloat16()
    wq = torch.randint(0, 256, (k // 2, n), dtype=torch.uint8, device="cuda", generator=g)
    s = (torch.rand(k // 128, n, device="cuda", generator=g) * 0.008 + 0.002).bfloat16()
    z = torch.randint(0, 16 if packed else 256, (k // 128, n), dtype=torch.uint8, device="cuda", generator=g)
    zp = z[:, 0::2] | (z[:, 1::2] << 4) if packed else z
    y = ops.w4a16_g128(x, wq, s, zp, zeros_packed=packed)
    q = torch.stack((wq & 15, wq >> 4), 1).reshape(k, n).double()
    zr, sr = (v.double().repeat_interleave(128, 0) for v in (z, s))
    ref, size = x.double() @ ((q - zr) * sr), x.double().abs() @ ((32 + q + zr) * sr)
    # an addition per 16 k, truncated, and the scale's product and sum per 128
    assert bool(((y.double() - ref).abs() <= 2.0 ** -8 * ref.abs() + (k // 16 + k // 64 + 16) * 2.0 ** -23 * size * 1.01).all())
    assert torch.equal(ops.w4a16_g128(x, wq, s, zp, zeros_packed=packed, static_weights=True), y)
