"""The int8 GEMM with K split over clusters, exactly, and the lines between it and the kernel for few rows."""

import pytest
import torch

from jax_metallib_b200 import ops

pytestmark = pytest.mark.gpu

# edges of row and column blocks, K of one stage, of ragged ones and of different lengths in a cluster, few and more blocks
# than a device holds clusters; both sides of the lines
SHAPES = [(33, 256, 512), (48, 4112, 272), (65, 4096, 1008), (128, 144, 4096), (129, 8192, 512), (200, 2064, 2304),
          (257, 16384, 256), (384, 1040, 1296), (512, 8192, 1024), (1000, 4096, 528), (64, 8192, 8192), (96, 4096, 6160),
          (32, 2048, 2048), (32, 2048, 2064), (17, 2064, 2048), (65, 512, 768), (193, 1024, 384), (193, 1024, 512)]


@pytest.mark.parametrize("a_unsigned,b_unsigned", [(False, False), (True, False), (False, True)])
@pytest.mark.parametrize("m,k,n", SHAPES)
def test_dots(cuda, m, k, n, a_unsigned, b_unsigned):
    g = torch.Generator(device="cuda").manual_seed(m + k + n)
    def codes(shape, unsigned):
        lo, hi, dtype = (0, 256, torch.uint8) if unsigned else (-128, 128, torch.int8)
        return torch.randint(lo, hi, shape, dtype=dtype, device="cuda", generator=g)
    a, b = codes((m, k), a_unsigned), codes((k, n), b_unsigned)
    row, col = torch.rand(m, device="cuda", generator=g), torch.rand(n, device="cuda", generator=g)
    ref = a.double() @ b.double()   # below 2^53: exact
    acc, out = ops.i8_dot(a, b, row, col)
    assert bool((acc.double() == ref).all())
    # the sum rounded to f32, then two products
    assert torch.equal(out, ref.float() * row[:, None] * col[None, :])
    assert torch.equal(ops.i8_dot(a, b, row, col, want_acc=False)[1], out)
