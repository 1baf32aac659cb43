"""int8 dots whose rows have no tensor map but are made of 8-byte pieces: copied asynchronously, a ring of stages ahead."""

import pytest
import torch

from jax_metallib_b200 import _lib, ops

pytestmark = pytest.mark.gpu


# one piece, whole and partial 16-byte pieces at the ends of rows and columns; K of one stage, of a part of one, of more than
# the ring holds; rows at the edges of the tiles of 8 to 64; tiles that change hands
@pytest.mark.parametrize("m,k,n", [(1, 8, 8), (3, 72, 24), (8, 64, 1000), (9, 1000, 136), (17, 4096, 120), (33, 328, 2056),
                                   (65, 2048, 1000), (70, 8, 4104), (17, 320, 124008), (1000, 328, 5000)])
@pytest.mark.parametrize("ta,tb,offset", [(torch.int8, torch.int8, 0), (torch.uint8, torch.int8, 8), (torch.int8, torch.uint8, 24)])
def test_pieces(cuda, m, k, n, ta, tb, offset):
    g = torch.Generator(device="cuda").manual_seed(m * k + n)

    def ints(rows, cols, t):
        lo = -128 if t == torch.int8 else 0
        flat = torch.randint(lo, lo + 256, (rows * cols + offset + 8,), dtype=torch.int16, device="cuda", generator=g).to(t)
        return flat[offset:offset + rows * cols].view(rows, cols)

    a, b = ints(m, k, ta), ints(k, n, tb)
    rs, cs = torch.rand(m, device="cuda", generator=g), torch.rand(n, device="cuda", generator=g)
    ref = (a.double() @ b.double()).to(torch.int64)
    for _ in range(2):
        acc, out = ops.i8_dot(a, b, rs, cs)
        assert torch.equal(acc.long(), ref) and torch.equal(out, ref.to(torch.int32).float() * rs[:, None] * cs)


@pytest.mark.parametrize("limit", [1, 5, 147])
def test_pieces_cta_limit(cuda, limit):
    g = torch.Generator(device="cuda").manual_seed(limit)
    a = torch.randint(-128, 128, (65, 1000), dtype=torch.int8, device="cuda", generator=g)
    b = torch.randint(-128, 128, (1000, 1000), dtype=torch.int8, device="cuda", generator=g)
    try:
        _lib.check(_lib.load().qmm_set_cta_limit(limit))
        acc = ops.i8_dot(a, b)[0]
    finally:
        _lib.check(_lib.load().qmm_set_cta_limit(0))
    assert torch.equal(acc.double(), a.double() @ b.double())
