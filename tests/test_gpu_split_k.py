"""The kernels that split K over a cluster, at the edges of their tiles, rings and routes, against 64-bit torch.

Tolerances: results are one rounding of a sum in f32.  A product is exact, so what is left beside that rounding is the sum's own
error, bounded by the number of additions on one element's path (truncated ones count twice) times 2^-24 of sum |x| |w|.
"""

import os
import subprocess
import sys

import pytest
import torch

from jax_metallib_b200 import _lib, ops, quantized

pytestmark = pytest.mark.gpu


def _gen(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    return g


def _sum_error(k, steps):
    """Additions: ``steps`` truncated ones in a stage of 64 k, one per stage after that, and sixteen partial tiles."""
    return (2 * steps + k / 64 + 16) * 2.0 ** -24


def _check(y, x, w, scale, rounding, steps):
    xd, wd = x.double(), w.double()
    ref, size = (xd @ wd) * scale, (xd.abs() @ wd.abs()) * scale.abs()
    bound = rounding * ref.abs() + _sum_error(x.shape[1], steps) * size * (1 + rounding)
    assert bool(((y.double() - ref).abs() <= bound).all()), ((y.double() - ref).abs() / bound.clamp_min(1e-300)).max().item()


@pytest.mark.parametrize("m,k,n", [(1, 8, 16), (1, 4096, 4096), (8, 72, 144), (9, 1032, 1040), (16, 4096, 28672), (17, 64, 128),
                                   (32, 4096, 28672), (33, 520, 272), (64, 14336, 256), (97, 1000, 5632),
                                   (97, 1000, 4736), (97, 2048, 5744), (1024, 248, 256), (1, 28672, 8192), (8, 33000, 16384)])
def test_int8_weights_bf16_rows(cuda, m, k, n):
    g = _gen(m + k + n)
    x = torch.randn(m, k, device="cuda", generator=g).bfloat16()
    w = torch.randint(-128, 128, (k, n), dtype=torch.int8, device="cuda", generator=g)
    s = torch.rand(n, device="cuda", generator=g) * 0.01 + 0.005
    # one accumulator runs over a CTA's slice of K, over 16 stages of 64 k (two warps share them) where a slice is longer than 64
    long = m <= 8 and k > 16384
    _check(ops.w8a16_perchannel(x, w, s), x, w, s.double(), 2.0 ** -8, 32 if long else k // 16 + 1)
    wide = torch.zeros(m, n + 32, dtype=torch.bfloat16, device="cuda")
    ops.w8a16_perchannel(x, w, s, out=wide, out_col_offset=16)
    assert torch.equal(wide[:, 16:16 + n], ops.w8a16_perchannel(x, w, s))
    assert not wide[:, :16].any() and not wide[:, 16 + n:].any()


@pytest.mark.parametrize("packed", [True, False])
@pytest.mark.parametrize("m,k,n", [(1, 128, 128), (8, 4096, 384), (9, 1280, 1536), (16, 14336, 256), (16, 384, 16384),
                                   (4, 6016, 12416), (5, 6144, 12416)])
def test_int4_weights(cuda, m, k, n, packed):
    g = _gen(m + k + n)
    x = (torch.randn(m, k, device="cuda", generator=g) * 3 + 1).bfloat16()
    x[0, 5] = 2e38 if packed else 2e37   # a product of the largest activations does not overflow where the result does not
    wq = torch.randint(0, 256, (k // 2, n), dtype=torch.uint8, device="cuda", generator=g)
    s = (torch.rand(k // 128, n, device="cuda", generator=g) * 0.008 + 0.002).bfloat16()
    z = torch.randint(0, 16 if packed else 256, (k // 128, n), dtype=torch.uint8, device="cuda", generator=g)
    zp = z[:, 0::2] | (z[:, 1::2] << 4) if packed else z
    y = ops.w4a16_g128(x, wq, s, zp, zeros_packed=packed)
    q = torch.stack((wq & 15, wq >> 4), 1).reshape(k, n).double()
    zr, sr = (v.double().repeat_interleave(128, 0) for v in (z, s))
    # the split kernel's products are x (q - z); the other one, which takes the large weights, takes z off afterwards
    size = (q - zr).abs() if 65536 <= n * k <= 75_000_000 else 32 + q + zr
    ref, size = x.double() @ ((q - zr) * sr), x.double().abs() @ (size * sr)
    assert bool(((y.double() - ref).abs() <= 2.0 ** -8 * ref.abs() + _sum_error(k, 4) * size * 1.01).all())


def test_int4_weights_behind_a_long_kernel(cuda):
    """A kernel that lets its successor start early and then runs for longer than the bounded waits (2 s) is no timeout."""
    lib, g = _lib.load(), _gen(3)
    a = torch.randint(-128, 128, (13000, 8193), dtype=torch.int8, device="cuda", generator=g)
    b = torch.randint(-128, 128, (8193, 16385), dtype=torch.int8, device="cuda", generator=g)
    x = torch.randn(8, 4096, device="cuda", generator=g).bfloat16()
    wq = torch.randint(0, 256, (2048, 4096), dtype=torch.uint8, device="cuda", generator=g)
    s = (torch.rand(32, 4096, device="cuda", generator=g) * 0.008 + 0.002).bfloat16()
    zp = torch.randint(0, 256, (32, 2048), dtype=torch.uint8, device="cuda", generator=g)
    y = ops.w4a16_g128(x, wq, s, zp, zeros_packed=True)
    begin, end = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    try:
        _lib.check(lib.qmm_set_cta_limit(1))   # one persistent CTA: the other SMs are free for the successor
        begin.record()
        ops.i8_dot(a, b)
    finally:
        _lib.check(lib.qmm_set_cta_limit(0))
    late = ops.w4a16_g128(x, wq, s, zp, zeros_packed=True)
    end.record()
    torch.cuda.synchronize()
    assert lib.qmm_device_status() == 0
    assert begin.elapsed_time(end) > 2200.0
    assert torch.equal(y, late)


@pytest.mark.parametrize("m,k,n", [(1, 4, 16), (8, 100, 48), (9, 64, 128), (17, 1024, 1024), (33, 4, 16), (100, 2052, 400),
                                   (256, 512, 144)])
def test_int8_weights_f32_rows(cuda, m, k, n):
    g = _gen(m + k + n)
    x = torch.randn(m, k, device="cuda", generator=g) * torch.exp2(torch.randint(-20, 20, (m, 1), device="cuda", generator=g))
    w = torch.randint(-128, 128, (k, n), dtype=torch.int8, device="cuda", generator=g)
    s = torch.rand(n, device="cuda", generator=g) * 0.01 + 0.005
    _check(ops.w8a32_perchannel(x, w, s), x, w, s.double(), 2.0 ** -22, 6)


@pytest.mark.parametrize("m,k,n", [(4, 96, 32), (8, 1024, 1024), (13, 260, 144), (40, 2048, 256)])
def test_int8_weights_f32_small_rows(cuda, m, k, n):
    """Activations down to the smallest f32, whole rows of them and among larger ones: no bit of them is lost."""
    g = _gen(m + k + n)
    w = torch.randint(-128, 128, (k, n), dtype=torch.int8, device="cuda", generator=g)
    scale = (torch.rand(n, device="cuda", generator=g) + 0.5) * 2.0 ** 100
    bits = torch.randn(m, k, device="cuda", generator=g).double()
    wd = w.double()
    for e in (-100, -109, -110, -111, -112, -118, -126, -133, -140, -148):
        mixed = torch.where(torch.rand(m, k, device="cuda", generator=g) < 0.1, e, -100)
        for x in ((bits * 2.0 ** e).float(), torch.ldexp(bits, mixed).float()):
            xd = x.double()
            y, ref, size = ops.w8a32_perchannel(x, w, scale).double(), (xd @ wd) * scale, (xd.abs() @ wd.abs()) * scale
            # beside the sum's own error, additions below 2^-126 round to 2^-149: one per stage of 32 k, and the partial tiles
            bound = 2.0 ** -22 * ref.abs() + _sum_error(k, 6) * size + (k / 32 + 20) * 2.0 ** -149 * scale
            assert bool(((y - ref).abs() <= bound).all()), (e, ((y - ref).abs() / bound).max().item())


def test_int8_weights_f32_special_values(cuda):
    x = torch.randn(5, 256, device="cuda", generator=_gen(1))
    x[0, 3], x[1, 7], x[2, 5], x[2, 9], x[3, 200] = float("inf"), float("nan"), -float("inf"), float("inf"), 1e36
    w = torch.randint(-128, 128, (256, 64), dtype=torch.int8, device="cuda", generator=_gen(2))
    y, ref = ops.w8a32_perchannel(x, w, torch.full((64,), 1e-3, device="cuda")), (x.double() @ w.double()) * 1e-3
    assert torch.equal(torch.isnan(y), torch.isnan(ref))
    assert torch.equal(torch.nan_to_num(y[0], nan=0.0), torch.nan_to_num(ref[0].float(), nan=0.0))
    _check(y[3:4], x[3:4], w, torch.tensor(1e-3, dtype=torch.float64, device="cuda"), 2.0 ** -22, 6)


@pytest.mark.parametrize("m", [1, 8, 9, 17, 33, 65])
@pytest.mark.parametrize("k,n", [(1, 1), (16, 17), (63, 65), (64, 128), (1000, 48), (331, 257), (2048, 1000)])
@pytest.mark.parametrize("ta,tb,offset", [(torch.int8, torch.int8, 0), (torch.uint8, torch.int8, 1), (torch.int8, torch.uint8, 3),
                                          (torch.uint8, torch.uint8, 2)])
def test_int8_dot_any_rows(cuda, m, k, n, ta, tb, offset):
    g = _gen(m * k + n)

    def ints(rows, cols, t):  # a view that begins `offset` bytes into its allocation
        lo = -128 if t == torch.int8 else 0
        flat = torch.randint(lo, lo + 256, (rows * cols + offset,), dtype=torch.int16, device="cuda", generator=g).to(t)
        return flat[offset:].view(rows, cols)

    a, b = ints(m, k, ta), ints(k, n, tb)
    rs, cs = torch.rand(m, device="cuda", generator=g), torch.rand(n, device="cuda", generator=g)
    acc, out = ops.i8_dot(a, b, rs, cs)
    ref = (a.double() @ b.double()).to(torch.int64)
    assert torch.equal(acc.long(), ref)
    assert torch.equal(out, ref.to(torch.int32).float() * rs[:, None] * cs)


# Three tiles and more to a cluster (296 CTAs are resident, 148 of the int8 dots' 64-row tiles): partial tiles change hands through
# buffers that come back, the rings run on over the tiles.
@pytest.mark.parametrize("m,k,n", [(3, 320, 124000), (16, 192, 124016), (32, 320, 124000), (31, 64, 115200)])
def test_tiles_change_hands_bf16_rows(cuda, m, k, n):
    g = _gen(m + k + n)
    w = torch.randint(-128, 128, (k, n), dtype=torch.int8, device="cuda", generator=g)
    s = torch.rand(n, device="cuda", generator=g) * 0.01 + 0.005
    for _ in range(4):
        x = torch.randn(m, k, device="cuda", generator=g).bfloat16()
        _check(ops.w8a16_perchannel(x, w, s), x, w, s.double(), 2.0 ** -8, k // 16 + 1)


@pytest.mark.parametrize("m,k,n", [(5, 320, 124000), (1000, 196, 2000)])
def test_tiles_change_hands_f32_rows(cuda, m, k, n):
    g = _gen(m + k + n)
    w = torch.randint(-128, 128, (k, n), dtype=torch.int8, device="cuda", generator=g)
    s = torch.rand(n, device="cuda", generator=g) * 0.01 + 0.005
    for _ in range(4):
        x = torch.randn(m, k, device="cuda", generator=g)
        _check(ops.w8a32_perchannel(x, w, s), x, w, s.double(), 2.0 ** -22, 6)


@pytest.mark.parametrize("m,k,n", [(8, 320, 124000), (16, 320, 124000), (32, 320, 124000), (1, 331, 124001), (17, 321, 124001),
                                   (1000, 331, 5001)])
def test_tiles_change_hands_int8_dot(cuda, m, k, n):
    g = _gen(m + k + n)
    b = torch.randint(-128, 128, (k, n), dtype=torch.int8, device="cuda", generator=g)
    for _ in range(4):
        a = torch.randint(-128, 128, (m, k), dtype=torch.int8, device="cuda", generator=g)
        assert torch.equal(ops.i8_dot(a, b)[0].double(), a.double() @ b.double())


@pytest.mark.parametrize("limit", [1, 5, 147])
def test_int8_dot_any_rows_cta_limit(cuda, limit):
    lib, g = _lib.load(), _gen(limit)
    a = torch.randint(-128, 128, (200, 331), dtype=torch.int8, device="cuda", generator=g)
    b = torch.randint(-128, 128, (331, 1001), dtype=torch.int8, device="cuda", generator=g)
    try:
        _lib.check(lib.qmm_set_cta_limit(limit))
        acc = ops.i8_dot(a, b)[0]
    finally:
        _lib.check(lib.qmm_set_cta_limit(0))
    assert torch.equal(acc.double(), a.double() @ b.double())


def _operator_weights(fmt, group, n, k, g):
    """Packed weights, call arguments and the dequantised weights [N, K] in 64 bits."""
    groups = (n, k // group)
    if fmt.startswith("affine"):
        bits = int(fmt[6:])
        q = torch.randint(0, 1 << bits, (n, k), device="cuda", generator=g)
        s = torch.rand(groups, device="cuda", generator=g) * 0.01 + 0.002
        b = -s * (1 << bits) / 2 * (0.9 + 0.2 * torch.rand(groups, device="cuda", generator=g))
        s[0], b[0], q[0] = 1.0, 0.04, 0    # a flat group
        packed = q.to(torch.uint8)
        if bits == 4:
            v = (q.view(n, k // 8, 8) << (4 * torch.arange(8, device="cuda"))).sum(-1)
            packed = torch.where(v >= 2 ** 31, v - 2 ** 32, v).to(torch.int32)
        w = s.double().repeat_interleave(group, 1) * q.double() + b.double().repeat_interleave(group, 1)
        size = s.double().repeat_interleave(group, 1) * q.double() + b.double().abs().repeat_interleave(group, 1)
        return lambda x: quantized.affine_quantized_matmul(x, packed, s, b, bits=bits, group_size=group, K=k), w, size
    if fmt == "mxfp8":
        packed = (torch.randn(n, k, device="cuda", generator=g) * 100).clamp(-448, 448).to(torch.float8_e4m3fn).view(torch.uint8)
        values = packed.view(torch.float8_e4m3fn).double()
    else:
        codes = torch.randint(0, 16, (n, k), dtype=torch.uint8, device="cuda", generator=g)
        packed = codes[:, 0::2] | (codes[:, 1::2] << 4)
        table = torch.tensor([0, .5, 1, 1.5, 2, 3, 4, 6], device="cuda", dtype=torch.float64)
        values = torch.cat((table, -table))[codes.long()]
    if fmt == "nvfp4":
        sb = (torch.rand(groups, device="cuda", generator=g) * 0.03 + 0.004).to(torch.float8_e4m3fn).view(torch.uint8)
        scale = sb.view(torch.float8_e4m3fn).double()
    else:
        sb = torch.randint(100, 123, groups, dtype=torch.uint8, device="cuda", generator=g)
        scale = torch.exp2(sb.double() - 127)
    w = values * scale.repeat_interleave(group, 1)
    return lambda x: quantized.quantized_matmul(x, packed, sb, mode=fmt, K=k), w, w.abs()


FORMATS = [("affine4", 32), ("affine4", 64), ("affine4", 96), ("affine4", 128), ("affine8", 32), ("affine8", 128), ("mxfp4", 32),
           ("mxfp8", 32), ("nvfp4", 16)]
# rows at the edges of the tiles of 32, 64 and 128; K of several boxes and of none; ragged columns
SHAPES = [(4, 384, 17), (17, 1152, 128), (33, 384, 200), (64, 2304, 130), (65, 1920, 333), (130, 5376, 260), (300, 1152, 96)]


def _check_operator(fmt, group, m, k, n, dtype):
    g = _gen(m + k + n)
    run, w, size = _operator_weights(fmt, group, n, k, g)
    x = torch.randn(m, k, device="cuda", generator=g).to(dtype)
    y, ref = run(x).double(), x.double() @ w.T
    # a unit of 64 k is twelve truncated additions (three terms), scaled, joined with its bias term and added in f32
    bound = (2.0 ** -11 if dtype == torch.float16 else 2.0 ** -24) * ref.abs() + _sum_error(k, 16) * (x.double().abs() @ size.T)
    if dtype == torch.float16:
        bound += 2.0 ** -24   # results below the smallest normal number
    assert bool(((y - ref).abs() <= bound).all()), (k, ((y - ref).abs() / bound).max().item())


@pytest.mark.parametrize("dtype", [torch.float16, torch.float32])
@pytest.mark.parametrize("m,k,n", SHAPES)
@pytest.mark.parametrize("fmt,group", FORMATS)
def test_operator_matmul(cuda, fmt, group, m, k, n, dtype):
    _check_operator(fmt, group, m, (k + group - 1) // group * group, n, dtype)


# Units of 32 k, an odd number of them: the last stage is half filled.  16384 columns leave one CTA to a tile, whose slice is all
# of K (1, 3, .. units, the last of them in every round of four or eight accumulators); 130 columns split K, and the last slice is odd.
HALF_STAGES = {16384: (32, 96, 160, 224, 288, 352, 416, 480, 544, 672, 800, 864), 130: (288, 1056, 1440, 2080, 2400)}


@pytest.mark.parametrize("dtype", [torch.float16, torch.float32])
@pytest.mark.parametrize("n", sorted(HALF_STAGES))
@pytest.mark.parametrize("m", [4, 48, 300])
@pytest.mark.parametrize("fmt,group", [("affine4", 32), ("affine4", 96), ("affine8", 32), ("affine8", 160), ("mxfp4", 32), ("mxfp8", 32)])
def test_operator_matmul_half_stage(cuda, fmt, group, m, n, dtype):
    widths = [k for k in HALF_STAGES[n] if k % group == 0 and k % 64 == 32]
    assert widths
    for k in widths:
        _check_operator(fmt, group, m, k, n, dtype)


@pytest.mark.parametrize("dtype", [torch.float16, torch.float32])
@pytest.mark.parametrize("fmt,group", [("affine4", 64), ("affine8", 32), ("mxfp4", 32), ("mxfp8", 32), ("nvfp4", 16)])
@pytest.mark.parametrize("m", [20, 70])
def test_operator_matmul_special_values(cuda, fmt, group, m, dtype):
    g = _gen(m)
    run, w, _ = _operator_weights(fmt, group, 160, 512, g)
    x = torch.randn(m, 512, device="cuda", generator=g)
    x[0, 5], x[1, 70], x[2, 100], x[2, 101], x[3, 400] = float("inf"), float("nan"), -float("inf"), float("inf"), -float("inf")
    x[4] = 1e-38 if dtype == torch.float32 else 6e-8
    x[5, 9] = 1e36 if dtype == torch.float32 else 6e4
    x = x.to(dtype)
    y, ref = run(x), x.double() @ w.T
    assert torch.equal(torch.isnan(y), torch.isnan(ref))
    assert torch.equal(torch.isinf(y[:4]), torch.isinf(ref[:4])) and torch.equal(torch.sign(y[0]), torch.sign(ref[0]).to(dtype))
    if dtype == torch.float32:
        size = x[5].double().abs() @ w.abs().T
        assert bool(((y[5].double() - ref[5]).abs() <= 2.0 ** -24 * ref[5].abs() + _sum_error(512, 64) * size).all())
        assert torch.allclose(y[4].double(), ref[4], rtol=1e-4, atol=512 * 2.0 ** -149)


@pytest.mark.parametrize("dtype", [torch.float16, torch.float32])
@pytest.mark.parametrize("fmt,group", [("affine4", 64), ("affine4", 32), ("affine8", 128)])
@pytest.mark.parametrize("m", [20, 70, 300])
def test_operator_matmul_infinite_weights(cuda, fmt, group, m, dtype):
    """Infinite scales and biases: weight by weight, an infinity times a code of 0 is NaN, and so are infinities of both signs."""
    g = _gen(m)
    n, k, bits = 160, 2048, int(fmt[6:])
    x = torch.randn(m, k, device="cuda", generator=g)
    x[0] = x[0].abs() + 0.01
    x = x.to(dtype)
    q = torch.randint(0, 1 << bits, (n, k), device="cuda", generator=g)
    q[4], q[8] = 3, 0
    s = torch.rand(n, k // group, device="cuda", generator=g) * 0.01 + 0.002
    b = torch.randn(n, k // group, device="cuda", generator=g) * 0.05
    s[3, 1], s[4, 1], b[5, 2], b[6, 3], s[8, 0], s[9, 2] = (float(v) for v in ("inf", "inf", "inf", "-inf", "inf", "nan"))
    packed = q.to(torch.uint8)
    if bits == 4:
        v = (q.view(n, k // 8, 8) << (4 * torch.arange(8, device="cuda"))).sum(-1)
        packed = torch.where(v >= 2 ** 31, v - 2 ** 32, v).to(torch.int32)
    y = quantized.affine_quantized_matmul(x, packed, s, b, bits=bits, group_size=group, K=k)
    ref = x.double() @ (s.double().repeat_interleave(group, 1) * q.double() + b.double().repeat_interleave(group, 1)).T
    assert torch.isinf(ref[0, 4:7]).all() and torch.isnan(ref[:, 8]).all() and torch.isnan(ref[1:, 5]).all()
    assert torch.equal(torch.isnan(y), torch.isnan(ref)) and torch.equal(torch.isinf(y), torch.isinf(ref))
    assert torch.equal(torch.sign(y)[torch.isinf(ref)], torch.sign(ref).to(dtype)[torch.isinf(ref)])
    finite = torch.isfinite(ref)
    assert ((y.double() - ref)[finite].norm() / ref[finite].norm()).item() < (1e-3 if dtype == torch.float16 else 1e-5)


@pytest.mark.parametrize("dtype", [torch.float16, torch.float32])
@pytest.mark.parametrize("fmt,group", [("mxfp4", 32), ("mxfp8", 32), ("nvfp4", 16)])
def test_operator_matmul_nan_codes(cuda, fmt, group, dtype):
    g = _gen(5)
    n, k = 40, 512
    x = torch.randn(20, k, device="cuda", generator=g).to(dtype)
    packed = torch.full((n, k if fmt == "mxfp8" else k // 2), 0x38 if fmt == "mxfp8" else 0x22, dtype=torch.uint8, device="cuda")
    scales = torch.full((n, k // group), 0x38 if fmt == "nvfp4" else 127, dtype=torch.uint8, device="cuda")
    scales[7, 3] = 0x7F if fmt == "nvfp4" else 0xFF
    if fmt == "mxfp8":
        packed[11, 200] = 0x7F
    y = quantized.quantized_matmul(x, packed, scales, mode=fmt, K=k)
    rows = torch.zeros(n, dtype=torch.bool, device="cuda")
    rows[[7, 11] if fmt == "mxfp8" else [7]] = True
    assert torch.equal(torch.isnan(y), rows.expand_as(y))


@pytest.mark.parametrize("call", [
    "ops.w8a16_perchannel(x.bfloat16(), w, s)", "ops.w8a32_perchannel(x, w, s)", "ops.i8_dot(w[:8], w.view(-1)[:1024 * 511].view(1024, 511))[0]",
    "quantized.affine_quantized_matmul(x, p, g, g, bits=4, group_size=64, K=1024)"])
def test_first_call_of_a_process_under_capture(cuda, call):
    """Nothing that a first call sets up (status word, attributes, occupancy) may break a capture that is under way."""
    program = f"""
import torch
from jax_metallib_b200 import _lib, ops, quantized
_lib.load()
x = torch.randn(8, 1024, device="cuda")
w = torch.randint(-127, 128, (1024, 1024), dtype=torch.int8, device="cuda")
s = torch.rand(1024, device="cuda")
p = torch.randint(-2**31, 2**31 - 1, (1024, 128), dtype=torch.int32, device="cuda")
g = torch.rand(1024, 16, device="cuda")
torch.cuda.synchronize()
graph = torch.cuda.CUDAGraph()
with torch.cuda.graph(graph):
    y = {call}
graph.replay()
torch.cuda.synchronize()
assert torch.equal(y, {call})
"""
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    subprocess.run([sys.executable, "-c", program], check=True, cwd=root, timeout=120)


def test_forced_routes(cuda):
    """The tests of this file once more with every shape on the kernels that split K or on the operator GEMM, small ones too."""
    if os.environ.get("QMM_FORCE_SPLIT_K"):
        pytest.skip("this is that run")
    subprocess.run([sys.executable, "-m", "pytest", "-q", "-x", "-m", "gpu", "-k", "not first_call and not long_kernel", __file__],
                   check=True, env=dict(os.environ, QMM_FORCE_SPLIT_K="1"), timeout=600)
