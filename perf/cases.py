"""What the speed of this framework is judged by.

Each case is one piece of work that a program built on this package hands it, called through the
public entry points: the StableHLO-level matmuls of ``ops``, the operator API of ``quantized``, the
captured decode step of ``decode_stack`` and a compiled program run through ``runtime``.  The matmuls
of a language model come as the four linears of one decoder layer (q|k|v, o, gate|up, down), as
``bench.py`` and ``decode_stack`` lay them out: no pass then finds its weights in L2 by accident.

``listed()`` names the cases, ``draw(rng)`` gives further ones over the same ranges.
"""

from __future__ import annotations

import math

import numpy as np
import torch

from jax_metallib_b200 import _lib, decode_stack, ops, quantized, runtime
from jax_metallib_b200.stablehlo import weight_only_linears_module

FORMATS = ("affine4", "affine8", "mxfp4", "mxfp8", "nvfp4")


def listed():
    return [
        # the smallest matmul of the package: int8 weights, f32 activations, one small dense layer
        {"name": "int8_f32_small", "op": "int8_f32", "m": 32, "k": 1024, "n": 1024},
        # a square int8 x int8 dot with its f32 rescale, prefill-sized
        {"name": "int8_dot_square", "op": "int8_dot", "m": 2048, "k": 4096, "n": 4096, "rescale": True},
        # a 1000-class head on a small batch: few rows, a column count that is no multiple of 16
        {"name": "int8_dot_head", "op": "int8_dot", "m": 65, "k": 2048, "n": 1000, "rescale": True},
        # decode of one sequence with int8 weights
        {"name": "int8_decode", "op": "int8_layer", "m": 1, "d": 4096, "kv": 1024, "ffn": 14336},
        # prefill with int8 weights at the width of a 70B-shaped layer: the headline of bench.py
        {"name": "int8_prefill", "op": "int8_layer", "m": 4096, "d": 8192, "kv": 1024, "ffn": 28672},
        # decode of a few sequences with int4 weights
        {"name": "int4_decode", "op": "int4_layer", "m": 4, "d": 4096, "kv": 1024, "ffn": 14336},
        # a prompt of odd length with int4 weights
        {"name": "int4_prefill_ragged", "op": "int4_layer", "m": 777, "d": 4096, "kv": 1024, "ffn": 14336},
        # a whole decode step as a captured graph: layers of an 8B-shaped model over its cache, and the lm_head.  Four layers:
        # the roundings between operators make two correct steps drift apart by 1.3 % over four layers, 4 % over 32
        {"name": "decode_step", "op": "decode_step", "batch": 8, "context": 2048, "layers": 4, "heads": 32, "kv_heads": 8,
         "ffn": 14336, "vocab": 32000},
        # operator API, decode of one sequence with half-precision activations
        {"name": "affine4_decode_f16", "op": "operator", "format": "affine4", "group": 64, "dtype": "f16", "m": 1, "d": 4096,
         "kv": 1024, "ffn": 14336},
        # operator API, a short prompt with single-precision activations (the default of the API)
        {"name": "affine4_prompt_f32", "op": "operator", "format": "affine4", "group": 64, "dtype": "f32", "m": 48, "d": 2048,
         "kv": 512, "ffn": 5632},
        # operator API, prefill with half-precision activations and an MX format
        {"name": "mxfp8_prefill_f16", "op": "operator", "format": "mxfp8", "group": 32, "dtype": "f16", "m": 512, "d": 4096,
         "kv": 1024, "ffn": 14336},
        # a compiled program of four linears run from host activations to host results
        {"name": "program_decode", "op": "program", "m": 8, "d": 4096, "kv": 1024, "ffn": 14336},
    ]


# ---------------------------------------------------------------------------
# more cases of the same ranges
# ---------------------------------------------------------------------------

def _log_int(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def _layer(rng, d_lo, d_hi, step=256):
    """Widths of a decoder layer: model width, key/value width, feed-forward width."""
    d = step * rng.randint(d_lo // step, d_hi // step)
    kv = max(128, d // rng.choice((4, 8)) // 128 * 128)
    ffn = int(d * rng.uniform(2.5, 3.5)) // step * step
    return {"d": d, "kv": kv, "ffn": ffn}


def draw(rng):
    op = rng.choice(("int8_f32", "int8_dot", "int8_dot", "int8_layer", "int8_layer", "int4_layer", "int4_layer", "decode_step",
                     "operator", "operator", "operator", "program"))
    if op == "int8_f32":
        k, n = _log_int(rng, 64, 4096), _log_int(rng, 64, 4096)
        if rng.random() < 0.75:
            k, n = max(16, k // 16 * 16), max(16, n // 16 * 16)
        return {"op": op, "m": _log_int(rng, 1, 256), "k": k, "n": n}
    if op == "int8_dot":
        k, n = _log_int(rng, 128, 8192), _log_int(rng, 128, 8192)
        if rng.random() < 0.67:
            k, n = k // 64 * 64, n // 64 * 64
        return {"op": op, "m": _log_int(rng, 1, 4096), "k": k, "n": n, "rescale": rng.random() < 0.75}
    if op == "int8_layer":
        return {"op": op, "m": _log_int(rng, 1, 3900), **_layer(rng, 1024, 8192)}
    if op == "int4_layer":
        return {"op": op, "m": _log_int(rng, 1, 3900), **_layer(rng, 1024, 8192)}
    if op == "decode_step":
        kv_heads = rng.choice((4, 8))
        heads = kv_heads * rng.choice((1, 2, 4))
        return {"op": op, "batch": _log_int(rng, 1, 16), "context": _log_int(rng, 100, 4000), "layers": rng.randint(1, 4),
                "heads": heads, "kv_heads": kv_heads, "ffn": heads * 128 * 7 // 2, "vocab": 64 * rng.randint(200, 1000)}
    if op == "operator":
        fmt = rng.choice(FORMATS)
        group = rng.choice((32, 64, 128)) if fmt.startswith("affine") else (16 if fmt == "nvfp4" else 32)
        dtype = rng.choice(("f16", "f16", "f32"))
        return {"op": op, "format": fmt, "group": group, "dtype": dtype, "m": _log_int(rng, 1, 500 if dtype == "f16" else 128),
                **_layer(rng, 1024, 4096)}
    return {"op": op, "m": _log_int(rng, 1, 512), **_layer(rng, 1024, 4096)}


def linears(case):
    """(K, N) of the four linears of the case's layer."""
    d, kv, ffn = case["d"], case["kv"], case["ffn"]
    return [(d, d + 2 * kv), (d, d), (d, 2 * ffn), (ffn, d)]


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------

def _gen(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    return g


def _normal(shape, gen, dtype):
    return torch.randn(shape, device="cuda", generator=gen, dtype=torch.float32).to(dtype)


def _uniform(shape, lo, hi, gen, dtype=torch.float32):
    return (torch.rand(shape, device="cuda", generator=gen) * (hi - lo) + lo).to(dtype)


def _int8(shape, gen):
    return torch.randint(-127, 128, shape, dtype=torch.int8, device="cuda", generator=gen)


def _activations(case, gen, dtype):
    """One activation tensor for each input width of the layer."""
    return {k: _normal((case["m"], k), gen, dtype) for k in (case["d"], case["ffn"])}


def _e2m1_codes(unit):
    """Nearest e2m1 code of values already divided by their scale."""
    mids = torch.tensor([0.25, 0.75, 1.25, 1.75, 2.5, 3.5, 5.0], device=unit.device)
    return torch.bucketize(unit.abs(), mids).to(torch.uint8) | ((unit < 0).to(torch.uint8) << 3)


def _operator_weights(fmt, group, n, k, gen):
    """Weights of a trained layer's spread, in the packing of the operator API."""
    g = k // group
    if fmt == "affine4":
        packed = torch.randint(-2**31, 2**31 - 1, (n, k // 8), dtype=torch.int32, device="cuda", generator=gen)
        scales = _uniform((n, g), 0.002, 0.006, gen)
        return {"packed": packed, "scales": scales, "biases": scales * -7.5 * _uniform((n, g), 0.9, 1.1, gen)}
    if fmt == "affine8":
        packed = torch.randint(0, 256, (n, k), dtype=torch.uint8, device="cuda", generator=gen)
        scales = _uniform((n, g), 0.0001, 0.0004, gen)
        return {"packed": packed, "scales": scales, "biases": scales * -127.5 * _uniform((n, g), 0.9, 1.1, gen)}
    if fmt == "mxfp8":
        packed = (_normal((n, k), gen, torch.float32) * 100).clamp_(-448, 448).to(torch.float8_e4m3fn).view(torch.uint8)
        return {"packed": packed, "scales": torch.randint(110, 115, (n, g), dtype=torch.uint8, device="cuda", generator=gen)}
    codes = _e2m1_codes(_normal((n, k), gen, torch.float32) * 2)
    packed = codes[:, 0::2] | (codes[:, 1::2] << 4)
    if fmt == "mxfp4":
        return {"packed": packed, "scales": torch.randint(118, 123, (n, g), dtype=torch.uint8, device="cuda", generator=gen)}
    return {"packed": packed, "scales": _uniform((n, g), 0.004, 0.03, gen, torch.float8_e4m3fn).view(torch.uint8)}


_client = None


def _runtime_client():
    """A program has one client for its life."""
    global _client
    if _client is None:
        _client = runtime.Client()
    return _client


def prepare(case, seed):
    op, gen = case["op"], _gen(seed)
    if op == "int8_f32":
        m, k, n = case["m"], case["k"], case["n"]
        return {"op": op, "x": _normal((m, k), gen, torch.float32), "w": _int8((k, n), gen), "s": _uniform((n,), 0.005, 0.02, gen)}
    if op == "int8_dot":
        m, k, n = case["m"], case["k"], case["n"]
        state = {"op": op, "a": _int8((m, k), gen), "b": _int8((k, n), gen), "row": None, "col": None}
        if case["rescale"]:
            state["row"], state["col"] = _uniform((m,), 0.01, 0.05, gen), _uniform((n,), 0.005, 0.02, gen)
        return state
    if op == "int8_layer":
        x = _activations(case, gen, torch.bfloat16)
        return {"op": op, "lins": [(x[k], _int8((k, n), gen), _uniform((n,), 0.005, 0.02, gen)) for k, n in linears(case)]}
    if op == "int4_layer":
        x = _activations(case, gen, torch.bfloat16)
        return {"op": op, "lins": [(x[k], decode_stack.random_int4_linear(k, n, 128, "cuda", gen)) for k, n in linears(case)]}
    if op == "decode_step":
        shape = decode_stack.LlamaShape(n_layers=case["layers"], d_model=case["heads"] * 128, n_heads=case["heads"],
                                        n_kv_heads=case["kv_heads"], ffn=case["ffn"], vocab=case["vocab"])
        b, ctx = case["batch"], case["context"]
        step = decode_stack.DecodeStep(shape, decode_stack.random_model(shape, "cuda", seed=seed), b, ctx, torch.device("cuda"))
        step.ids.copy_(torch.randint(0, shape.vocab, (b,), dtype=torch.int32, device="cuda", generator=gen))
        kc, vc = ([_normal((b, shape.n_kv_heads, ctx, 128), gen, torch.bfloat16) for _ in range(shape.n_layers)] for _ in range(2))
        torch.cuda.synchronize()
        step.capture(kc, vc)
        return {"op": op, "step": step, "kc": kc, "vc": vc}
    if op == "operator":
        x = _activations(case, gen, torch.float16 if case["dtype"] == "f16" else torch.float32)
        lins = [(x[k], k, _operator_weights(case["format"], case["group"], n, k, gen)) for k, n in linears(case)]
        return {"op": op, "format": case["format"], "group": case["group"], "lins": lins}
    client = _runtime_client()
    shapes = linears(case)
    exe = client.compile(weight_only_linears_module([(case["m"], k, n, 1 if k == case["ffn"] else 0) for k, n in shapes]))
    x = [_normal((case["m"], k), gen, torch.bfloat16).cpu().view(torch.int16).numpy().view(np.uint16) for k in (case["d"], case["ffn"])]
    weights = []
    for k, n in shapes:
        w, s = _int8((k, n), gen), _uniform((n,), 0.005, 0.02, gen)
        weights.append(client.view_of_device_memory(w.data_ptr(), _lib.QMM_S8, w.shape, keepalive=w))
        weights.append(client.view_of_device_memory(s.data_ptr(), _lib.QMM_F32, s.shape, keepalive=s))
    torch.cuda.synchronize()
    return {"op": op, "client": client, "exe": exe, "x": x, "weights": weights}


# ---------------------------------------------------------------------------
# one pass
# ---------------------------------------------------------------------------

def run(state):
    op = state["op"]
    if op == "int8_f32":
        return ops.w8a32_perchannel(state["x"], state["w"], state["s"])
    if op == "int8_dot":
        acc, out = ops.i8_dot(state["a"], state["b"], state["row"], state["col"], want_acc=state["row"] is None)
        return acc if out is None else out
    if op == "int8_layer":
        return [ops.w8a16_perchannel(x, w, s) for x, w, s in state["lins"]]
    if op == "int4_layer":
        return [ops.w4a16_g128(x, lin["wq"], lin["s"], lin["z"], zeros_packed=True, static_weights=True) for x, lin in state["lins"]]
    if op == "decode_step":
        step = state["step"]
        step.graph.replay()
        return [step.logits, step.new_k, step.new_v]
    if op == "operator":
        fmt = state["format"]
        if fmt.startswith("affine"):
            return [quantized.affine_quantized_matmul(x, w["packed"], w["scales"], w["biases"], bits=int(fmt[6:]),
                                                      group_size=state["group"], K=k) for x, k, w in state["lins"]]
        return [quantized.quantized_matmul(x, w["packed"], w["scales"], mode=fmt, K=k) for x, k, w in state["lins"]]
    client = state["client"]
    x = [client.buffer_from_host(a, dtype=_lib.QMM_BF16) for a in state["x"]]
    outs, _done = state["exe"].execute(x + state["weights"])
    return [torch.from_numpy(y.to_numpy().view(np.int16)).view(torch.bfloat16) for y in outs]


# ---------------------------------------------------------------------------
# what a pass cannot do without, and how far correct results may lie apart
# ---------------------------------------------------------------------------

def work(case):
    op = case["op"]
    if op == "int8_f32":
        m, k, n = case["m"], case["k"], case["n"]
        return {"bytes": k * n + 4 * (m * k + n + m * n), "flops": 2 * m * k * n}
    if op == "int8_dot":
        m, k, n = case["m"], case["k"], case["n"]
        return {"bytes": m * k + k * n + 4 * m * n + (4 * (m + n) if case["rescale"] else 0), "flops": 2 * m * k * n}
    if op == "decode_step":
        shape = decode_stack.LlamaShape(n_layers=case["layers"], d_model=case["heads"] * 128, n_heads=case["heads"],
                                        n_kv_heads=case["kv_heads"], ffn=case["ffn"], vocab=case["vocab"])
        weights = sum(k * n for k, n in shape.linears().values()) * shape.n_layers + shape.d_model * shape.vocab
        attention = 2 * shape.n_heads * 128 * (case["context"] + 1) * shape.n_layers
        new = 2 * 2 * case["layers"] * case["batch"] * case["kv_heads"] * 128
        return {"bytes": shape.weight_bytes_per_step(case["batch"], case["context"]) + 2 * case["batch"] * case["vocab"] + new,
                "flops": 2 * case["batch"] * (weights + attention)}
    m, shapes = case["m"], linears(case)
    act = 4 if case.get("dtype") == "f32" else 2
    total = act * m * (case["d"] + case["ffn"] + sum(n for _, n in shapes))
    for k, n in shapes:
        if op == "int4_layer":
            total += k * n // 2 + k // 128 * n * 5 // 2
        elif op == "operator":
            bits = 8 if case["format"] in ("affine8", "mxfp8") else 4
            total += k * n * bits // 8 + k // case["group"] * n * (8 if case["format"].startswith("affine") else 1)
        else:
            total += k * n + 4 * n
    return {"bytes": total, "flops": 2 * m * sum(k * n for k, n in shapes)}


def tolerance(case):
    """About four times the distance (2-norm) of the results from the same matmul in 64 bits."""
    op = case["op"]
    if op == "int8_dot":
        return "exact"  # integers, and one f32 rounding for each of the two multiplies in their stated order
    if op == "int8_f32" or case.get("dtype") == "f32":
        return {"rel": 1e-5}  # 4e-7 for sums split over a warp, some 2e-6 for one sum running over all of K = 14336
    if op == "operator":
        return {"rel": 1e-3}  # 2.1e-4: one rounding to f16
    if op == "decode_step":
        return {"rel": 3e-2}  # 0.4 to 1.3 % over one to four layers with a rounding to bf16 after every operator
    return {"rel": 1e-2}  # 1.7e-3 for one rounding to bf16, 2.3e-3 where the dequantised weights are rounded to bf16 too


# ---------------------------------------------------------------------------
# the same results in 64 bits, by torch alone
# ---------------------------------------------------------------------------

def _int4_weights(lin):
    """(q - z) * s of one int4 linear: [K, N]."""
    wq, z = lin["wq"], lin["z"]
    q = torch.stack((wq & 15, wq >> 4), dim=1).reshape(-1, wq.shape[1]).double()
    zero = torch.stack((z & 15, z >> 4), dim=2).reshape(z.shape[0], -1).double()
    return (q - zero.repeat_interleave(128, 0)) * lin["s"].double().repeat_interleave(128, 0)


_E2M1 = (0.0, 0.5, 1.0, 1.5, 2.0, 3.0, 4.0, 6.0)


def _operator_dequantised(fmt, group, w):
    """Weights of the operator API's formats: [N, K]."""
    packed, n = w["packed"], w["packed"].shape[0]
    if fmt == "affine4":
        values = torch.stack([(packed >> (4 * j)) & 15 for j in range(8)], dim=2).reshape(n, -1).double()
    elif fmt == "affine8":
        values = packed.double()
    elif fmt == "mxfp8":
        values = packed.view(torch.float8_e4m3fn).float().double()
    else:
        table = torch.tensor(_E2M1 + tuple(-v for v in _E2M1), dtype=torch.float64, device=packed.device)
        values = table[torch.stack((packed & 15, packed >> 4), dim=2).reshape(n, -1).long()]
    if fmt.startswith("affine"):
        scale = w["scales"].double()
    elif fmt == "nvfp4":
        scale = w["scales"].view(torch.float8_e4m3fn).float().double()
    else:
        scale = torch.exp2(w["scales"].double() - 127)
    values = (values.reshape(n, -1, group) * scale[:, :, None]).reshape(n, -1)
    return values + w["biases"].double().repeat_interleave(group, 1) if fmt.startswith("affine") else values


def _exact_decode_step(state):
    step = state["step"]
    shape, model, b = step.shape, step.model, step.B
    hq, hkv, hd = shape.n_heads, shape.n_kv_heads, shape.head_dim

    def norm(h, w):
        return h * torch.rsqrt(h.square().mean(-1, keepdim=True) + shape.eps) * w.double()

    angle = step.pos.double()[:, None] * shape.rope_theta ** (-2.0 * torch.arange(hd // 2, device="cuda", dtype=torch.float64) / hd)
    cos, sin = torch.cos(angle)[:, None], torch.sin(angle)[:, None]

    def rope(t):
        lo, hi = t[..., :hd // 2], t[..., hd // 2:]
        return torch.cat((lo * cos - hi * sin, hi * cos + lo * sin), -1)

    h = model["embed"][step.ids.long()].double()
    keys, values = [], []
    for layer, kc, vc in zip(model["layers"], state["kc"], state["vc"]):
        n = norm(h, layer["attn_norm"])
        q, k, v = ((n @ _int4_weights(layer[name])).reshape(b, -1, hd) for name in "qkv")
        q, k = rope(q), rope(k)
        keys.append(k.reshape(b, -1))
        values.append(v.reshape(b, -1))
        p = torch.softmax(q.reshape(b, hkv, hq // hkv, hd) @ torch.cat((kc.double(), k[:, :, None]), 2).mT / hd ** 0.5, -1)
        h = h + (p @ torch.cat((vc.double(), v[:, :, None]), 2)).reshape(b, -1) @ _int4_weights(layer["o"])
        n = norm(h, layer["mlp_norm"])
        h = h + (torch.nn.functional.silu(n @ _int4_weights(layer["gate"])) * (n @ _int4_weights(layer["up"]))) @ _int4_weights(layer["down"])
    return [norm(h, model["final_norm"]) @ model["lm_head"].double(), torch.stack(keys), torch.stack(values)]


def exact(case, seed):
    """What ``run`` returns for the inputs of ``prepare(case, seed)``, in 64 bits."""
    if case["op"] == "program":  # its weights lie in the runtime's buffers: drawn again, in prepare's order
        gen = _gen(seed)
        x = {k: _normal((case["m"], k), gen, torch.bfloat16) for k in (case["d"], case["ffn"])}
        outs = []
        for k, n in linears(case):
            w, s = _int8((k, n), gen), _uniform((n,), 0.005, 0.02, gen)
            outs.append(((x[k].double() @ w.double()) * s.double()).cpu())
        return outs
    state = prepare(case, seed)
    op = state["op"]
    if op == "int8_f32":
        return state["x"].double() @ state["w"].double() * state["s"].double()
    if op == "int8_dot":
        acc = state["a"].double() @ state["b"].double()
        return acc if state["row"] is None else acc * state["row"].double()[:, None] * state["col"].double()
    if op == "int8_layer":
        return [x.double() @ w.double() * s.double() for x, w, s in state["lins"]]
    if op == "int4_layer":
        return [x.double() @ _int4_weights(lin) for x, lin in state["lins"]]
    if op == "decode_step":
        return _exact_decode_step(state)
    return [x.double() @ _operator_dequantised(state["format"], state["group"], w).T for x, _, w in state["lins"]]
