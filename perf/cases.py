"""What the quantized layer is asked to do: the cases that its speed is measured on.

Three kinds of program use this package: a serving loop that calls ``MixedQLinear`` layers (decode with few tokens, prompts of
every length), a decoder block that wires seven of them with its norms, attention and MLP, and a program that calls the
operators of the extension one by one.  ``listed`` names points of that range and ``draw`` gives others of it.

The layer shapes of the listed cases are those of one Llama-2 decoder layer (``quik_b200.workloads``); weights and activations
follow the same distributions: weights N(0, 0.02) on a per-channel grid, activations N(0, 1) with the outlier columns x20.
"""
from __future__ import annotations

import copy
import functools
import math

import torch

from quik_b200 import asymmetric, matmul
from quik_b200.block import QuikLlamaBlock
from quik_b200.qlinear import MixedQLinear, pack_to_i4

DTYPES = {"float16": torch.float16, "bfloat16": torch.bfloat16}
# one decoder layer, fused-N shapes: "in x out x bits" per linear layer (down_proj runs in 8 bits)
LAYERS_7B = "4096x12288x4 4096x4096x4 4096x22016x4 11008x4096x8"
LAYERS_70B = "8192x10240x4 8192x8192x4 8192x57344x4 28672x8192x8"


def listed():
    return [
        # the smallest call: one token through one 4096 x 4096 layer, bound by latency, launches and host work
        _layers("linear_1_token", "4096x4096x4", 1, "float16", 256, False),
        # decode steps: the linear layers of one decoder layer for a batch of sequences, one token each
        _layers("decode_7b_16_tokens", LAYERS_7B, 16, "float16", 256, False),
        _layers("decode_70b_5_tokens_bf16", LAYERS_70B, 5, "bfloat16", 256, False),
        # a larger decode batch, or the last piece of a chunked prompt
        _layers("batch_7b_96_tokens", LAYERS_7B, 96, "float16", 256, False),
        # short prompts, of no particular length
        _layers("prompt_7b_333_tokens", LAYERS_7B, 333, "float16", 256, False),
        # a prompt of one full context, the setting of the layer benchmarks
        _layers("prompt_7b_2048_tokens", LAYERS_7B, 2048, "float16", 256, False),
        # the largest: a long prompt through the largest model's layers
        _layers("prompt_70b_4096_tokens", LAYERS_70B, 4096, "float16", 256, False),
        # a layer as it is converted from a model with biases, at sizes that fill no tile
        _layers("linear_odd_bias_bf16", "5152x7000x8 5152x3333x4", 741, "bfloat16", 96, True),
        # whole decoder blocks: fused producers, shared quantized inputs, rotary embedding, attention, residuals
        _block("block_7b_2048_tokens", 2048, 4096, 32, 32, 11008, "float16"),
        _block("block_gqa_77_tokens_bf16", 77, 4096, 32, 8, 11008, "bfloat16"),
        # the operators one by one, as a program written for the extension calls them
        _ops("operators_4bit_2048_tokens", 4, 2048, 4096, 4096, 256, "float16"),
        # the 8-bit operators at a ragged size, with the fused product + dequantize operator
        _ops("operators_8bit_777_tokens", 8, 777, 3008, 5000, 64, "float16"),
    ]


def draw(rng):
    """One more case of the same ranges; sizes log-uniform, most of them no multiple of a tile."""
    def log_between(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    def multiple(lo, hi, of):
        return max(1, round(log_between(lo, hi) / of)) * of

    kind = rng.choice(["layers"] * 7 + ["block", "ops", "ops"])
    dtype = rng.choice(["float16", "float16", "bfloat16"])
    while True:
        if kind == "block":
            heads = rng.choice([8, 16, 32])
            return _block(None, log_between(1, 2048), 128 * heads, heads, rng.choice([heads, heads // 4]),
                          multiple(256 * heads, 448 * heads, 64), dtype)
        if kind == "ops":
            bits = rng.choice([4, 8])
            case = _ops(None, bits, log_between(16, 4096), multiple(1024, 12288, 32), log_between(1000, 24000),
                        rng.choice([0, 64, 128, 256]), dtype if bits == 4 else "float16")
        else:
            shapes = ["%dx%dx%d" % (multiple(1024, 28672, 32), rng.choice([log_between(1024, 57344), multiple(1024, 57344, 128)]),
                                    rng.choice([4, 4, 4, 8])) for _ in range(rng.choice([1, 2, 4]))]
            case = _layers(None, " ".join(shapes), log_between(1, 4096), dtype, rng.choice([0, 64, 128, 256, 256, 256, 368, 512]),
                           rng.random() < 0.3)
        if work(case)["flops"] <= 2e12 and work(case)["bytes"] <= 1.2e9:
            return case


# ---- case descriptions ------------------------------------------------------------------------------------------------------
def _named(name, case):
    return case if name is None else {"name": name, **case}


def _layers(name, shapes, tokens, dtype, outliers, bias):
    return _named(name, {"kind": "layers", "shapes": shapes, "tokens": tokens, "dtype": dtype, "outliers": outliers,
                         "bias": bias})


def _block(name, tokens, hidden, heads, kv_heads, intermediate, dtype):
    return _named(name, {"kind": "block", "tokens": tokens, "hidden": hidden, "heads": heads, "kv_heads": kv_heads,
                         "intermediate": intermediate, "dtype": dtype, "outliers": 256})


def _ops(name, bits, tokens, k, n, outliers, dtype):
    return _named(name, {"kind": "ops", "bits": bits, "tokens": tokens, "k": k, "n": n, "outliers": outliers, "dtype": dtype})


def _shapes(case):
    return [tuple(int(v) for v in s.split("x")) for s in case["shapes"].split()]


def _block_shapes(case):
    h, kv, i = case["hidden"], case["hidden"] // case["heads"] * case["kv_heads"], case["intermediate"]
    return [(h, kv, 4), (h, kv, 4), (h, h, 4), (h, h, 4), (h, i, 4), (h, i, 4), (i, h, 8)]


# ---- inputs and weights -----------------------------------------------------------------------------------------------------
def _codes(n, k, bits, gen):
    """Weight codes of N(0, 0.02) weights: the grid step is 0.02 / 2.6 (4 bits) or 0.02 / 40 (8 bits)."""
    lo, hi = (-8, 7) if bits == 4 else (-128, 127)
    step = 2.6 if bits == 4 else 40.0
    return torch.randn(n, k, device="cuda", generator=gen).mul_(step).round_().clamp_(lo, hi).to(torch.int8)


def _fill(layer, gen, columns=None):
    """Random weights of the layer's own format, on the GPU; ``columns``: (integer, outlier) column ids to use."""
    n, k, f, bits = layer.out_features, layer.in_features, layer.fp_features_num, layer.bits
    codes = _codes(n, k - f, bits, gen)
    scale = (0.02 / (2.6 if bits == 4 else 40.0)) * (0.9 + 0.2 * torch.rand(n, 1, device="cuda", generator=gen))
    layer.int_weight.copy_(pack_to_i4(codes) if bits == 4 else codes)
    layer.weights_scales.copy_(scale)
    layer.reduced_w.copy_((codes.sum(1, dtype=torch.float32) * scale[:, 0]).reshape(1, n))
    if f:
        layer.fp_weight.copy_(0.02 * torch.randn(n, f, device="cuda", generator=gen))
    if layer.bias is not None:
        layer.bias.copy_(0.1 * torch.randn(n, device="cuda", generator=gen))
    if columns is not None:
        layer.int_indices.copy_(columns[0])
        layer.fp_indices.copy_(columns[1])


def _columns(k, f, gen):
    perm = torch.randperm(k, device="cuda", generator=gen)
    return torch.sort(perm[f:])[0], torch.sort(perm[:f])[0]


def _activations(rows, k, outlier_ids, dtype, gen):
    x = torch.randn(rows, k, device="cuda", generator=gen)
    x[:, outlier_ids] *= 20
    return x.to(dtype)


@functools.lru_cache(maxsize=2)
def _block_template(hidden, heads, kv_heads, intermediate, dtype, outliers):
    """The block's construction (weights drawn and quantized on the host) costs seconds: it is done once per shape, the
    weights are then drawn anew on the GPU for every state."""
    return QuikLlamaBlock(hidden=hidden, heads=heads, kv_heads=kv_heads, intermediate=intermediate, bits=4, down_bits=8,
                          fp_features=outliers, dtype=DTYPES[dtype], clip=False)


def prepare(case, seed):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    dtype, f, m = DTYPES[case["dtype"]], case["outliers"], case["tokens"]
    state = {"kind": case["kind"]}
    if case["kind"] == "layers":
        state["layers"] = []
        for k, n, bits in _shapes(case):
            with torch.device("cuda"):
                layer = MixedQLinear(k, n, fp_features_num=f, bits=bits, dtype=dtype)
            if not case["bias"]:
                layer.bias = None
            columns = _columns(k, f, gen)
            _fill(layer, gen, columns)
            state["layers"].append((layer, _activations(m, k, columns[1], dtype, gen).unsqueeze(0)))
    elif case["kind"] == "block":
        block = copy.deepcopy(_block_template(case["hidden"], case["heads"], case["kv_heads"], case["intermediate"],
                                              case["dtype"], f))
        for layer in block.modules():
            if isinstance(layer, MixedQLinear):
                _fill(layer, gen)
        for norm in (block.input_norm, block.post_norm):
            norm.copy_(1 + 0.1 * torch.randn(norm.shape, device="cuda", generator=gen))
        state["block"] = block
        # the residual stream of a trained model is several times one block's update (RMSNorm takes the factor out again)
        state["x"] = 8 * _activations(m, case["hidden"], block.q_proj.fp_indices, dtype, gen).unsqueeze(0)
    else:
        k, n, bits = case["k"], case["n"], case["bits"]
        codes = _codes(n, k - f, bits, gen)
        scale = ((0.02 / (2.6 if bits == 4 else 40.0)) * (0.9 + 0.2 * torch.rand(n, device="cuda", generator=gen)))
        state.update(
            bits=bits, int_ids=None, w=pack_to_i4(codes) if bits == 4 else codes, scale=scale.to(dtype).reshape(n, 1),
            reduced=(codes.sum(1, dtype=torch.float32) * scale).to(dtype).reshape(1, n),
            fp_w=(0.02 * torch.randn(n, f, device="cuda", generator=gen)).to(dtype))
        state["int_ids"], state["fp_ids"] = _columns(k, f, gen)
        state["x"] = _activations(m, k, state["fp_ids"], dtype, gen)
    return state


def run(state):
    if state["kind"] == "layers":
        return [layer(x) for layer, x in state["layers"]]
    if state["kind"] == "block":
        with torch.no_grad():
            return state["block"](state["x"])
    s = state
    bits = s["bits"]
    codes, meta, fp_x = asymmetric.quantize(s["x"], s["int_ids"], s["fp_ids"], bits)
    y = torch.nn.functional.linear(fp_x, s["fp_w"])
    if bits == 4:
        acc = matmul.int4Matmul(codes, s["w"])
        return {"codes": codes, "meta": meta, "fp_x": fp_x, "acc": acc,
                "out": asymmetric.dequantize(acc, meta, s["scale"], s["reduced"], y, bits)}
    scale_row, zero_row = meta.view(-1, 2).t().contiguous()
    return {"codes": codes, "meta": meta, "fp_x": fp_x, "acc": matmul.int8Matmul(codes, s["w"]),
            "out": asymmetric.int8FusedDequantize(codes, s["w"], scale_row, s["scale"], 128.0, zero_row, s["reduced"], y)}


# ---- what a pass cannot do without, and how exact it is ---------------------------------------------------------------------
def _layer_work(m, k, n, bits, f, bias=False):
    """Weights in their storage format, 16-bit activations in and out, per-channel vectors."""
    return ((k - f) * n * bits / 8 + 2 * f * n + (6 if bias else 4) * n + 2 * m * (k + n), 2.0 * m * n * k)


def work(case):
    m, f = case["tokens"], case["outliers"]
    if case["kind"] == "layers":
        parts = [_layer_work(m, k, n, bits, f, case["bias"]) for k, n, bits in _shapes(case)]
    elif case["kind"] == "block":
        h, kv, i = case["hidden"], case["hidden"] // case["heads"] * case["kv_heads"], case["intermediate"]
        # the weights once and the block's own input and output; the products and causal attention
        parts = [(_layer_work(0, k, n, bits, f)[0], 2.0 * m * n * k) for k, n, bits in _block_shapes(case)]
        parts.append((4.0 * m * h, 2.0 * m * m * h))
    else:
        k, n, bits = case["k"], case["n"], case["bits"]
        codes = m * (k - f) * bits / 8
        # each operator reads its inputs and writes its outputs: quantize, product, linear, dequantize (8 bits: the fused form)
        parts = [(2 * m * k + codes + 2 * m * f, 0.0), (codes + n * (k - f) * bits / 8 + 4 * m * n, 2.0 * m * n * (k - f)),
                 (2 * f * (m + n) + 2 * m * n, 2.0 * m * n * f)]
        parts.append((8 * m * n, 0.0) if bits == 4 else (codes + n * (k - f) + 4 * m * n, 2.0 * m * n * (k - f)))
    return {"bytes": float(sum(p[0] for p in parts)), "flops": float(sum(p[1] for p in parts))}


def tolerance(case):
    """Four times what the path differs from itself in 64 bits.  A layer differs by its 16-bit roundings: 2.9e-4 (float16) and
    2.3e-3 (bfloat16) of the result's norm; codes and integer sums are exact.  In a block every quantizer turns a rounding
    of its input into a step of the 4-bit grid where a value lies next to a boundary, which makes 2.6e-3 (float16) to 4.3e-3
    (bfloat16) of the output, and up to 0.083 of its root mean square in one value."""
    if case["kind"] == "block":
        return {"rel": 1.7e-2, "max": 0.34}
    return {"rel": 1.2e-3 if case["dtype"] == "float16" else 1e-2}
