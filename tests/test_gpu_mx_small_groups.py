"""MX matmuls whose weights hold groups far below the largest scale of their 512 k: what f16 cannot hold beside it is added in f32,
group by group, and costs little.

Tolerance: that of the other MX prefill sums (an accumulator takes 32 truncated additions in a unit of 512 k, units and up to eight
slices are added in f32, one rounding to f16), and for the groups 32 additions each and one for each group of the column.
"""

import pytest
import torch

from jax_metallib_b200 import quantized

pytestmark = pytest.mark.gpu

BITS = {"mxfp4": 4, "mxfp8": 8}


def _values(mode, packed, scales):
    if mode == "mxfp8":
        values = packed.view(torch.float8_e4m3fn).double()
    else:
        table = torch.tensor([0, .5, 1, 1.5, 2, 3, 4, 6], device="cuda", dtype=torch.float64)
        codes = torch.stack((packed & 15, packed >> 4), 2).flatten(1).long()
        values = torch.cat((table, -table))[codes]
    return values * torch.exp2(scales.double() - 127).repeat_interleave(32, 1)


def _weights(mode, n, k, g, lo, hi):
    if mode == "mxfp8":
        packed = (torch.randn(n, k, device="cuda", generator=g) * 100).clamp(-448, 448).to(torch.float8_e4m3fn).view(torch.uint8)
    else:
        packed = torch.randint(0, 256, (n, k // 2), dtype=torch.uint8, device="cuda", generator=g)
    return packed, torch.randint(lo, hi, (n, k // 32), dtype=torch.uint8, device="cuda", generator=g)


# K in slices and whole, tiles of 16 to 192 rows, scales that come in pieces of 16 bytes and one by one
@pytest.mark.parametrize("m,k,n", [(9, 2048, 160), (33, 1056, 257), (100, 14336, 200), (129, 1536, 9600), (150, 1024, 19200), (385, 608, 6401)])
@pytest.mark.parametrize("mode", sorted(BITS))
def test_added(cuda, mode, m, k, n):
    """Activations are zero where the scales are large: the results of every third column are the small groups'."""
    g = torch.Generator(device="cuda").manual_seed(m)
    packed, scales = _weights(mode, n, k, g, 170, 176)
    scales[1::3], scales[2::3] = 100, 122   # columns without such groups
    x = torch.zeros(m, k, device="cuda", dtype=torch.half)
    for group in (0, 5, 17, 18, k // 32 - 1):
        scales[::3, group] = torch.randint(120, 126, (len(scales[::3]),), dtype=torch.uint8, device="cuda", generator=g)
        x[:, 32 * group:32 * group + 32] = torch.randn(m, 32, device="cuda", generator=g).half() / 8
    w = _values(mode, packed, scales)
    y = quantized.quantized_matmul(x, packed, scales, mode=mode, K=k).double()
    ref, size = x.double() @ w.T, x.double().abs() @ w.abs().T
    bound = 2.0 ** -11 * ref.abs() + 2.0 ** -24 + (2 * 32 + k / 32 + 48) * 2.0 ** -24 * size
    assert bool(((y - ref).abs() <= bound).all()), ((y - ref).abs() / bound).max().item()
    assert bool((y[:, ::3].abs().amax(0) > 0).all())


@pytest.mark.parametrize("m,k,n", [(24, 2048, 160), (100, 1024, 130), (150, 1024, 19200)])
@pytest.mark.parametrize("mode", sorted(BITS))
def test_not_finite(cuda, mode, m, k, n):
    """An infinity that meets a small group is one in the result, and a NaN where the weight is zero."""
    g = torch.Generator(device="cuda").manual_seed(m)
    packed, scales = _weights(mode, n, k, g, 110, 116)
    scales[:, 4] = 60
    x = torch.randn(m, k, device="cuda", generator=g).half()
    x[1, 130], x[7, 140], x[m - 1, 159], x[3, 700] = float("inf"), float("-inf"), float("nan"), float("inf")
    y = quantized.quantized_matmul(x, packed, scales, mode=mode, K=k)
    w = _values(mode, packed, scales)
    for row, at in ((1, 130), (7, 140), (3, 700)):
        want = x[row, at].double() * w[:, at]
        assert torch.equal(y[row].isnan(), want.isnan()) and torch.equal(y[row][~want.isnan()].double(), want[~want.isnan()])
    assert bool(y[m - 1].isnan().all())
    rows = [r for r in range(m) if r not in (1, 7, 3, m - 1)]
    assert bool(y[rows].isfinite().all())


def _time(call, n=10):
    call()
    start, stop = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    best = float("inf")
    for _ in range(3):
        torch.cuda.synchronize()
        start.record()
        for _ in range(n):
            call()
        stop.record()
        torch.cuda.synchronize()
        best = min(best, start.elapsed_time(stop) / n)
    return best


@pytest.mark.parametrize("mode", sorted(BITS))
def test_cost(cuda, mode):
    """Two such groups in every 16th column do not double the time (a column computed again by one thread: 30 ms)."""
    m, k, n = 512, 14336, 4096
    g = torch.Generator(device="cuda").manual_seed(1)
    packed, scales = _weights(mode, n, k, g, 110, 116)
    x = torch.randn(m, k, device="cuda", generator=g).half()
    plain = _time(lambda: quantized.quantized_matmul(x, packed, scales, mode=mode, K=k))
    scales[::16, 40], scales[::16, 300] = 60, 60
    assert _time(lambda: quantized.quantized_matmul(x, packed, scales, mode=mode, K=k)) < 2 * plain
