"""The work this library is measured by: quantized linears, the projections of a dense decoder block and sparse-MoE
expert layers, each called the way a host program calls them, over the sizes such programs reach.

  linear   one `QuantMethod.forward`: a single projection (an attention output, a vocabulary head)
  block    the projections of one dense decoder block in their order: fused QKV where the three formats agree (else
           three calls), attention output, fused gate/up, down
  moe      one sparse-MoE layer from router logits to the layer's output: the one-call layer with 16-bit activations
           (`forward_layer`), or with 8-bit activations (`act8`) router + `forward_fp8_act` / `forward_mx_act`, the
           shared expert included where the layer has one

Shapes are those of this repository's benchmark configurations (Llama-3-8B, Qwen3-30B-A3B, DeepSeek-V3 and gpt-oss-120b
layers); `draw` spreads rows, features, experts and formats over the same ranges.  Weights are N(0, 0.02^2) quantized to
the format, activations and logits N(0, 1), all made on the GPU from the seed."""
from __future__ import annotations

import math

import torch

import engine_b200 as hq
from engine_b200 import _lib as L

# GGML type -> (weights per block, bytes per block, byte offsets of the block's f16 fields)
GGML = {"Q8_0": (32, 34, (0,)), "Q4_K": (256, 144, (0, 2)), "Q6_K": (256, 210, (208,)), "Q5_K": (256, 176, (0, 2)),
        "Q4_0": (32, 18, (0,)), "Q5_0": (32, 22, (0,)), "Q4_1": (32, 20, (0, 2)), "Q5_1": (32, 24, (0, 2)),
        "Q2_K": (256, 84, (80, 82)), "Q3_K": (256, 110, (108,))}
DTYPES = {"f32": torch.float32, "f16": torch.float16, "bf16": torch.bfloat16}
CHUNK = 1 << 25      # weights quantized at a time


def listed():
    block = {"kind": "block", "hidden": 4096, "kv": 1024, "inter": 14336, "dtype": "bf16"}
    q4k = {"kind": "moe", "format": "Q4_K", "experts": 128, "top_k": 8, "hidden": 2048, "inter": 768, "act8": False}
    mx = {"kind": "moe", "format": "MXFP4", "experts": 128, "top_k": 4, "hidden": 2880, "inter": 2880}
    return [
        # the smallest call: one square projection for one token, weights small enough to stay in L2
        {"name": "linear_q4k_1row", "kind": "linear", "format": "Q4_K", "n": 4096, "k": 4096, "m": 1, "dtype": "f32"},
        # single-stream decode of an 8B dense model, one block
        {"name": "block_q8_0_1row", "format": "Q8_0", "m": 1, **block},
        # four streams of the usual 4-bit file, which keeps `attn_v` and `ffn_down` in Q6_K
        {"name": "block_q4km_4rows", "format": "Q4_K_M", "m": 4, **block},
        # the vocabulary head over a full decode batch
        {"name": "head_q8_0_8rows", "kind": "linear", "format": "Q8_0", "n": 128256, "k": 4096, "m": 8, "dtype": "bf16"},
        # a serving batch of 32 streams on a block-FP8 checkpoint
        {"name": "block_fp8_32rows", "format": "FP8", "m": 32, **block},
        # a prompt of odd length
        {"name": "block_q4km_777rows", "format": "Q4_K_M", "m": 777, **block},
        # single-stream MoE decode: launches count
        {"name": "moe_q4k_1token", "tokens": 1, **q4k},
        # a decode batch that touches nearly every expert with a few rows each
        {"name": "moe_q4k_64tokens", "tokens": 64, **q4k},
        # a batch of prompts
        {"name": "moe_q4k_4096tokens", "tokens": 4096, **q4k},
        # MXFP4 decode batch, 16-bit activations
        {"name": "moe_mxfp4_128tokens", "tokens": 128, "act8": False, **mx},
        # MXFP4 prompts on the block-scaled MMA
        {"name": "moe_mxfp4_8192tokens", "tokens": 8192, "act8": True, **mx},
        # the largest: 11 GB of block-FP8 experts plus the shared expert, 8-bit activations
        {"name": "moe_fp8_4096tokens", "kind": "moe", "format": "FP8", "experts": 256, "top_k": 8, "hidden": 7168,
         "inter": 2048, "tokens": 4096, "act8": True},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _draw_linear(rng):
    fmt = rng.choice(["Q4_K", "Q6_K", "Q8_0", "FP8"] * 3 + ["Q5_K", "Q4_0", "Q5_0", "Q4_1", "Q5_1", "Q2_K", "Q3_K", "MXFP4"])
    k = 256 * _log(rng, 4, 56)
    n = _log(rng, 512, 131072)
    if fmt == "FP8":                       # checkpoints cut features in multiples of 64 (latent projections) or 128
        n = 64 * max(8, n // 64)
    m = _log(rng, 1, 4096)
    while m * n * k > 3e11:                # a share of the largest listed case
        m = max(1, m // 2)
        n = n if m > 8 else max(512, n // 2)
    if fmt == "FP8":
        n = 64 * max(8, n // 64)
    return {"kind": "linear", "format": fmt, "n": n, "k": k, "m": m, "dtype": rng.choice(["bf16", "bf16", "f16", "f32"])}


def _draw_block(rng):
    hidden = 512 * rng.randint(4, 10)
    return {"kind": "block", "format": rng.choice(["Q8_0", "Q4_K_M", "FP8"]), "hidden": hidden,
            "kv": hidden // rng.choice([2, 4]), "inter": 256 * rng.randint(hidden // 100, hidden // 70),
            "m": _log(rng, 1, 2048), "dtype": rng.choice(["bf16", "bf16", "f16"])}


def _draw_moe(rng):
    fmt = rng.choice(["Q4_K", "MXFP4", "FP8"])
    case = {"kind": "moe", "format": fmt, "tokens": _log(rng, 1, 4096)}
    if fmt == "Q4_K":
        case.update(experts=rng.choice([32, 64, 96, 128]), top_k=rng.randint(2, 8), hidden=256 * rng.randint(6, 16),
                    inter=256 * rng.randint(2, 8), act8=False)
    elif fmt == "MXFP4":
        case.update(experts=rng.choice([32, 64, 128]), top_k=4, hidden=64 * rng.randint(24, 56),
                    inter=64 * rng.randint(24, 48), act8=rng.random() < 0.5)
    else:
        case.update(experts=rng.choice([32, 64, 128, 160]), top_k=rng.randint(4, 8), hidden=512 * rng.randint(6, 14),
                    inter=512 * rng.randint(1, 4), act8=rng.random() < 0.75)
    return case


def draw(rng):
    return rng.choice([_draw_linear, _draw_linear, _draw_block, _draw_moe, _draw_moe])(rng)


# ---- inputs ------------------------------------------------------------------------------------------------------

def _u8(t):
    return t.contiguous().view(torch.uint8).reshape(*t.shape[:-1], t.shape[-1] * t.element_size())


def _weights(blocks, size, gen):
    return torch.randn((blocks, size), generator=gen, device="cuda") * 0.02


def _q8_0(blocks, gen):
    w = _weights(blocks, 32, gen)
    d = w.abs().amax(1, keepdim=True) / 127.0
    return torch.cat([_u8(d.half()), _u8((w / d).round().to(torch.int8))], 1)


def _q4_k(blocks, gen):
    w = _weights(blocks * 8, 32, gen).view(blocks, 8, 32)
    low = w.amin(2).clamp(max=0.0)
    step = (w.amax(2) - low) / 15.0
    d, dmin = (step.amax(1, keepdim=True) / 63.0).half(), (-low.amin(1, keepdim=True) / 63.0).half()
    sc = (step / d.float()).round().clamp(0, 63)
    mn = (-low / dmin.float().clamp_min(1e-12)).round().clamp(0, 63)
    q = ((w + (dmin.float() * mn).unsqueeze(2)) / (d.float() * sc).clamp_min(1e-12).unsqueeze(2)).round_().clamp_(0, 15)
    q, sc, mn = q.to(torch.uint8), sc.to(torch.uint8), mn.to(torch.uint8)
    packed = torch.cat([sc[:, :4] | ((sc[:, 4:] >> 4) << 6), mn[:, :4] | ((mn[:, 4:] >> 4) << 6),
                        (sc[:, 4:] & 15) | ((mn[:, 4:] & 15) << 4)], 1)
    return torch.cat([_u8(d), _u8(dmin), packed, (q[:, 0::2] | (q[:, 1::2] << 4)).reshape(blocks, 128)], 1)


def _q6_k(blocks, gen):
    w = _weights(blocks * 16, 16, gen).view(blocks, 16, 16)
    step = w.abs().amax(2) / 31.0
    d = (step.amax(1, keepdim=True) / 127.0).half()
    sc = (step / d.float()).round().clamp(1, 127)
    q = ((w / (d.float() * sc).unsqueeze(2)).round_().clamp_(-32, 31) + 32).to(torch.uint8).view(blocks, 2, 4, 32)
    low = torch.cat([q[:, :, 0] & 15 | ((q[:, :, 2] & 15) << 4), q[:, :, 1] & 15 | ((q[:, :, 3] & 15) << 4)], 2)
    high = (q[:, :, 0] >> 4) | ((q[:, :, 1] >> 4) << 2) | ((q[:, :, 2] >> 4) << 4) | ((q[:, :, 3] >> 4) << 6)
    return torch.cat([low.reshape(blocks, 128), high.reshape(blocks, 64), sc.to(torch.uint8), _u8(d)], 1)


def _ggml_other(fmt):
    """Blocks of the less common GGML types: every byte pattern is a valid block once its f16 fields are set."""
    weights, size, fields = GGML[fmt]

    def make(blocks, gen):
        raw = torch.randint(0, 256, (blocks, size), generator=gen, device="cuda", dtype=torch.uint8)
        for at in fields:
            scale = 2.0 ** -11 * (0.5 + torch.rand((blocks, 1), generator=gen, device="cuda"))
            raw[:, at:at + 2] = _u8((-8 * scale if at == 2 and weights == 32 else scale).half())
        return raw
    return make


def _ggml(fmt, e, n, k, gen):
    weights, size, _ = GGML[fmt]
    make = {"Q8_0": _q8_0, "Q4_K": _q4_k, "Q6_K": _q6_k}.get(fmt) or _ggml_other(fmt)
    out = torch.empty((e * n * k // weights, size), dtype=torch.uint8, device="cuda")
    step = CHUNK // weights
    for at in range(0, out.shape[0], step):
        out[at:at + step] = make(min(step, out.shape[0] - at), gen)
    return out.view(e, n, k // weights * size)


def _fp8(e, n, k, gen):
    nb = -(-n // 128)
    codes = torch.empty((e, nb * 128, k), dtype=torch.uint8, device="cuda")
    scales = torch.empty((e * nb, k // 128), device="cuda")
    rows = codes.view(e * nb, 128, k)
    step = max(1, CHUNK // (128 * k))
    for at in range(0, e * nb, step):
        count = min(step, e * nb - at)
        w = _weights(count * 128, k, gen).view(count, 128, k // 128, 128)
        s = w.abs().amax((1, 3)) / 448.0
        w /= s[:, None, :, None]
        rows[at:at + count] = w.to(torch.float8_e4m3fn).view(torch.uint8).view(count, 128, k)
        scales[at:at + count] = s
    return codes[:, :n].contiguous(), scales.view(e, nb, k // 128)


def _mxfp4(e, n, k, gen):
    blocks = torch.empty((e * n * k // 32, 16), dtype=torch.uint8, device="cuda")
    scales = torch.empty((e * n * k // 32,), dtype=torch.uint8, device="cuda")
    edges = torch.tensor([0.25, 0.75, 1.25, 1.75, 2.5, 3.5, 5.0], device="cuda")
    step = CHUNK // 32
    for at in range(0, blocks.shape[0], step):
        w = _weights(min(step, blocks.shape[0] - at), 32, gen)
        exp = torch.floor(torch.log2(w.abs().amax(1) / 6.0))
        q = torch.bucketize(w.abs() / torch.exp2(exp)[:, None], edges, out_int32=True).to(torch.uint8)
        q |= (w < 0).to(torch.uint8) << 3
        blocks[at:at + step] = q[:, 0::2] | (q[:, 1::2] << 4)
        scales[at:at + step] = (exp + 127).to(torch.uint8)
    return blocks.view(e, n, k // 2), scales.view(e, n, k // 32)


def _layer(fmt, n, k, gen, experts=0, bias=False):
    """One quantized projection, or a bank of `experts` of them."""
    e = max(1, experts)
    pick = (lambda t: t) if experts else (lambda t: t[0])
    b = (torch.randn((e, n), generator=gen, device="cuda") * 0.02).bfloat16() if bias else None
    if fmt == "FP8":
        codes, scales = _fp8(e, n, k, gen)
        return hq.BlockwiseFP8Linear(pick(codes), pick(scales), b)
    if fmt == "MXFP4":
        blocks, scales = _mxfp4(e, n, k, gen)
        return hq.MXFP4Layer(pick(blocks), pick(scales), b)
    return hq.GgufMatMul(pick(_ggml(fmt, e, n, k, gen)), fmt, k, b)


def _parts(case):
    """The projections of a block: (name, format, features out, features in)."""
    h, kv, inter, fmt = case["hidden"], case["kv"], case["inter"], case["format"]
    main, wide = ("Q4_K", "Q6_K") if fmt == "Q4_K_M" else (fmt, fmt)
    return [("q", main, h, h), ("k", main, kv, h), ("v", wide, kv, h), ("o", main, h, h), ("gate", main, inter, h),
            ("up", main, inter, h), ("down", wide, h, inter)]


def prepare(case, seed):
    gen = torch.Generator(device="cuda")
    gen.manual_seed(int(seed))

    def normal(rows, cols, dtype=torch.float32):
        return torch.randn((rows, cols), generator=gen, device="cuda").to(dtype)

    state = {"case": case}
    if case["kind"] == "linear":
        state["layer"] = _layer(case["format"], case["n"], case["k"], gen)
        state["x"] = normal(case["m"], case["k"], DTYPES[case["dtype"]])
    elif case["kind"] == "block":
        for name, fmt, n, k in _parts(case):
            state[name] = _layer(fmt, n, k, gen)
        state["x"] = normal(case["m"], case["hidden"], DTYPES[case["dtype"]])
        state["attn"] = normal(case["m"], case["hidden"], DTYPES[case["dtype"]])
    else:
        e, h, i, fmt = case["experts"], case["hidden"], case["inter"], case["format"]
        if fmt == "MXFP4":       # interleaved gate/up rows with biases, softmax over the chosen experts
            state["experts"] = hq.MoEExperts(_layer(fmt, h, i, gen, e, True), gate_up_proj=_layer(fmt, 2 * i, h, gen, e, True),
                                             act=L.ACT_GPTOSS, limit=7.0, alpha=1.702)
            state["router"] = hq.MoeRouterTopKConfig(case["top_k"], L.SCORE_RAW, L.WEIGHT_SOFTMAX, False)
        else:
            state["experts"] = hq.MoEExperts(_layer(fmt, h, i, gen, e), _layer(fmt, i, h, gen, e), _layer(fmt, i, h, gen, e))
            state["router"] = hq.MoeRouterTopKConfig(case["top_k"], L.SCORE_SOFTMAX, L.WEIGHT_SCORE, True)
        state["bias"] = None
        if fmt == "FP8":         # sigmoid scores, a selection bias, and with 8-bit activations the shared expert
            state["router"] = hq.MoeRouterTopKConfig(case["top_k"], L.SCORE_SIGMOID, L.WEIGHT_SCORE, True, 1e-20, 2.5)
            state["bias"] = torch.randn(e, generator=gen, device="cuda") * 0.01
            if case["act8"]:
                state["shared"] = hq.MoEExperts(_layer(fmt, h, i, gen, 1), _layer(fmt, i, h, gen, 1), _layer(fmt, i, h, gen, 1))
        state["x"] = normal(case["tokens"], h, torch.bfloat16)
        state["logits"] = normal(case["tokens"], e)
    return state


# ---- one pass ------------------------------------------------------------------------------------------------------

def run(state):
    case, x = state["case"], state["x"]
    if case["kind"] == "linear":
        return state["layer"].forward(x)
    if case["kind"] == "block":
        qkv = hq.try_fused_quantized_qkv(x, state["q"], state["k"], state["v"])
        if qkv is None:
            qkv = tuple(state[name].forward(x) for name in ("q", "k", "v"))
        hidden = state["o"].forward(state["attn"])
        inter = hq.try_fused_quantized_gate_up(hidden, state["gate"], state["up"])
        return {"q": qkv[0], "k": qkv[1], "v": qkv[2], "hidden": hidden, "inter": inter, "out": state["down"].forward(inter)}
    experts, logits = state["experts"], state["logits"]
    if not case["act8"]:
        return experts.forward_layer(x, logits, state["router"], state["bias"])
    top = hq.moe_router_topk(logits, state["router"], state["bias"])
    if case["format"] == "MXFP4":
        return experts.forward_mx_act(x, top.values, top.indices)
    return experts.forward_fp8_act(x, top.values, top.indices, shared_out=state["shared"].forward_fp8_dense(x))


# ---- what a pass cannot do without ---------------------------------------------------------------------------------

def _weight_bytes(fmt, n, k):
    if fmt == "FP8":
        return n * k + -(-n // 128) * (k // 128) * 4
    if fmt == "MXFP4":
        return n * k // 2 + n * k // 32
    weights, size, _ = GGML[fmt]
    return n * k // weights * size


def work(case):
    if case["kind"] == "linear":
        n, k, m = case["n"], case["k"], case["m"]
        size = DTYPES[case["dtype"]].itemsize
        return {"bytes": _weight_bytes(case["format"], n, k) + size * m * (n + k), "flops": 2 * m * n * k}
    if case["kind"] == "block":
        h, kv, inter, m = case["hidden"], case["kv"], case["inter"], case["m"]
        parts = _parts(case)
        size = DTYPES[case["dtype"]].itemsize
        return {"bytes": sum(_weight_bytes(fmt, n, k) for _, fmt, n, k in parts) + size * m * (2 * h + 3 * h + 2 * kv + inter),
                "flops": 2 * m * sum(n * k for _, _, n, k in parts)}
    e, h, i, t, k, fmt = (case[key] for key in ("experts", "hidden", "inter", "tokens", "top_k", "format"))
    touched = e * (1.0 - (1.0 - k / e) ** t)                # experts that at least one token chose, on average
    expert = 2 * _weight_bytes(fmt, i, h) + _weight_bytes(fmt, h, i) + (2 * (2 * i + h) if fmt == "MXFP4" else 0)
    shared = 1 if fmt == "FP8" and case["act8"] else 0
    return {"bytes": int((touched + shared) * expert) + t * (4 * h + 4 * e), "flops": 6 * t * (k + shared) * h * i}


def tolerance(case):
    """16-bit outputs: their own rounding, and a flip of the last bit of a 16-bit (or, with 8-bit activations, of an
    8-bit) intermediate.  32-bit outputs: the activations or the expanded weights are held in 16 bits."""
    if case["kind"] == "linear" and case["dtype"] == "f32":
        return {"rel": 1e-3}
    if case["kind"] != "moe" and case["dtype"] == "f16":
        return {"rel": 2e-3}
    return {"rel": 1e-2}
