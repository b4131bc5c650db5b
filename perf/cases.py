"""Performance cases of the block-FP8 path, from one decode token to a large prefill.

Four kinds of call, each through the entry point a model uses:

* linear: a quantised linear layer (`ReplicatedLinear`, `ColumnParallelLinear`) on 16-bit activations;
* mlp:    gate_up (column) -> fused silu * up + re-quantisation -> down (row), as a dense transformer block runs it;
* moe:    routing on the router's logits, then `FusedMoE` over all experts;
* quant:  the activation quantizer on its own.

Decode batches of a MoE layer may be replayed from a CUDA graph, as servers do.
"""
from __future__ import annotations

import math

import torch

from sglang_b200 import ops
from sglang_b200.srt.layers.linear import (
    ColumnParallelLinear,
    MergedColumnParallelLinear,
    ReplicatedLinear,
    RowParallelLinear,
)
from sglang_b200.srt.layers.moe.fused_moe_triton.layer import FusedMoE
from sglang_b200.srt.layers.moe.token_dispatcher import StandardTopKOutput
from sglang_b200.srt.layers.moe.topk import biased_grouped_topk, fused_topk
from sglang_b200.srt.layers.quantization.fp8 import Fp8Config
from sglang_b200.srt.layers.quantization.fp8_kernel import per_token_group_quant_fp8

DEV = "cuda"
DTYPES = {"bf16": torch.bfloat16, "fp16": torch.float16, "fp32": torch.float32}
WEIGHT_STD = 0.02


def listed():
    return [
        # one decoded token through DeepSeek-V3's fused q_a / kv_a projection: launches and latency
        {"name": "linear_decode_1", "kind": "linear", "m": 1, "n": 2112, "k": 7168, "dtype": "bf16", "bias": False},
        # a small square layer at a decode batch
        {"name": "linear_64_square", "kind": "linear", "m": 64, "n": 4096, "k": 4096, "dtype": "bf16", "bias": False},
        # a decode batch through DeepSeek-V3's widest dense layer: weight streaming
        {"name": "linear_64_gate_up", "kind": "linear", "m": 64, "n": 36864, "k": 7168, "dtype": "bf16", "bias": False},
        # Llama-3-70B's qkv projection on a ragged chunk of tokens, with a bias, in float16
        {"name": "linear_257_qkv", "kind": "linear", "m": 257, "n": 10240, "k": 8192, "dtype": "fp16", "bias": True},
        # prefill through DeepSeek-V3's kv_b: a short K and a wide output
        {"name": "linear_4096_kv_b", "kind": "linear", "m": 4096, "n": 32768, "k": 512, "dtype": "bf16", "bias": False},
        # prefill through DeepSeek-V3's gate_up: the largest dense product
        {"name": "linear_4096_gate_up", "kind": "linear", "m": 4096, "n": 36864, "k": 7168, "dtype": "bf16", "bias": False},
        # one GPU's eighth of Llama-3-70B's MLP on an odd number of tokens
        {"name": "mlp_1999", "kind": "mlp", "m": 1999, "h": 8192, "i": 3584, "dtype": "bf16"},
        # Qwen3-30B-A3B's MoE layer on a decode batch, replayed from a CUDA graph
        {"name": "moe_qwen_32_graph", "kind": "moe", "m": 32, "e": 128, "topk": 8, "h": 2048, "i": 768, "skew": 0.0,
         "gate": "softmax", "graph": True, "dtype": "bf16"},
        # the same layer on a large prefill with Zipf-skewed routing
        {"name": "moe_qwen_16384_skewed", "kind": "moe", "m": 16384, "e": 128, "topk": 8, "h": 2048, "i": 768,
         "skew": 1.2, "gate": "softmax", "graph": False, "dtype": "bf16"},
        # DeepSeek-V3's routed experts on a decode batch: most experts get a few rows each
        {"name": "moe_deepseek_64", "kind": "moe", "m": 64, "e": 256, "topk": 8, "h": 7168, "i": 2048, "skew": 0.0,
         "gate": "grouped", "graph": False, "dtype": "bf16"},
        # the same on a prefill: the largest case
        {"name": "moe_deepseek_4096", "kind": "moe", "m": 4096, "e": 256, "topk": 8, "h": 7168, "i": 2048, "skew": 0.0,
         "gate": "grouped", "graph": False, "dtype": "bf16"},
        # the quantizer alone on a long prefill, scales in the M-major layout
        {"name": "quant_8192", "kind": "quant", "m": 8192, "k": 18432, "column_major": True, "dtype": "bf16"},
    ]


def _log_int(rng, lo, hi, step=1):
    """An integer in [lo, hi], spread over the logarithm, rounded to a multiple of `step`."""
    v = math.exp(rng.uniform(math.log(lo), math.log(hi)))
    return min(hi, max(lo, int(round(v / step)) * step))


def _draw_once(rng):
    kind = rng.choices(["linear", "mlp", "moe", "quant"], [5, 2, 3, 1])[0]
    dtype = rng.choice(["bf16", "bf16", "fp16"])
    if kind == "linear":
        return {"kind": kind, "m": _log_int(rng, 1, 8192), "n": _log_int(rng, 512, 36864, rng.choice([8, 64, 128])),
                "k": _log_int(rng, 512, 18432, 128), "dtype": dtype, "bias": rng.random() < 0.25}
    if kind == "mlp":
        return {"kind": kind, "m": _log_int(rng, 1, 8192), "h": _log_int(rng, 1024, 8192, 128),
                "i": _log_int(rng, 512, 28672, 128), "dtype": dtype}
    if kind == "quant":
        return {"kind": kind, "m": _log_int(rng, 1, 16384), "k": _log_int(rng, 512, 18432, 128),
                "column_major": rng.random() < 0.5, "dtype": rng.choice(["bf16", "fp16", "fp32"])}
    m, e = _log_int(rng, 1, 16384), rng.choice([8, 16, 32, 64, 128, 256])
    return {"kind": kind, "m": m, "e": e, "topk": rng.randint(1, min(8, e // 2)),
            "h": _log_int(rng, 1024, 7168, 128), "i": _log_int(rng, 256, 2048, 128),
            "skew": rng.choice([0.0, 0.6, 1.2]), "gate": rng.choice(["softmax", "grouped"]),
            "graph": m <= 256 and rng.random() < 0.5, "dtype": dtype}


def _cost(case):
    w = work(case)
    return max(w["bytes"], w["flops"] / 50)


def draw(rng):
    most = max(_cost(c) for c in listed())
    while True:
        case = _draw_once(rng)
        if _cost(case) <= most:
            return case


# ---- inputs ---------------------------------------------------------------------------------------------------------


def _fill_codes(dst, gen):
    """Codes of N(0, 0.02) weights quantised per 128 x 128 block: the block's largest of 16384 values (about four
    standard deviations) lands on 448."""
    flat = dst.view(-1)
    step = 1 << 28
    for b in range(0, flat.numel(), step):
        part = flat[b : b + step]
        part.copy_(torch.randn(part.shape, generator=gen, device=DEV, dtype=torch.bfloat16).mul_(110.0).clamp_(-448.0, 448.0))


def _fill_scales(dst, gen):
    dst.copy_(torch.rand(dst.shape, generator=gen, device=DEV).mul_(0.2).add_(0.9).mul_(WEIGHT_STD / 110.0))


def _fill_layer(layer, gen):
    _fill_codes(layer.weight.data, gen)
    _fill_scales(layer.weight_scale_inv.data, gen)
    if layer.bias is not None:
        layer.bias.data.copy_(torch.randn(layer.bias.shape, generator=gen, device=DEV))
    return layer


def _activations(m, k, dtype, gen):
    """Hidden states with a few channels that are an order of magnitude larger than the rest."""
    x = torch.randn(m, k, generator=gen, device=DEV)
    hot = torch.randint(0, k, (max(1, k // 256),), generator=gen, device=DEV)
    x[:, hot] *= 10.0
    return x.to(dtype)


def _router_logits(case, gen):
    """Logits whose top-k follows a Zipf law of exponent `skew` over the experts (0 = uniform)."""
    m, e = case["m"], case["e"]
    popularity = -case["skew"] * torch.log(torch.arange(1, e + 1, device=DEV, dtype=torch.float32))
    popularity = popularity[torch.randperm(e, generator=gen, device=DEV)]
    noise = -torch.log(-torch.log(torch.rand(m, e, generator=gen, device=DEV).clamp_(1e-6, 1 - 1e-6)))
    return noise + popularity


def prepare(case, seed):
    gen = torch.Generator(device=DEV).manual_seed(seed)
    dtype = DTYPES[case["dtype"]]
    kind = case["kind"]
    cfg = Fp8Config()
    if kind == "quant":
        return {"case": case, "x": _activations(case["m"], case["k"], dtype, gen)}
    if kind == "linear":
        if case["bias"] or case["n"] % 128 == 0:
            layer = ColumnParallelLinear(case["k"], case["n"], bias=case["bias"], params_dtype=dtype, quant_config=cfg,
                                         device=DEV)
        else:
            layer = ReplicatedLinear(case["k"], case["n"], params_dtype=dtype, quant_config=cfg, device=DEV)
        return {"case": case, "x": _activations(case["m"], case["k"], dtype, gen), "layer": _fill_layer(layer, gen)}
    if kind == "mlp":
        gate_up = MergedColumnParallelLinear(case["h"], [case["i"], case["i"]], params_dtype=dtype, quant_config=cfg,
                                             device=DEV)
        down = RowParallelLinear(case["i"], case["h"], params_dtype=dtype, quant_config=cfg, device=DEV)
        return {"case": case, "x": _activations(case["m"], case["h"], dtype, gen), "gate_up": _fill_layer(gate_up, gen),
                "down": _fill_layer(down, gen)}
    moe = FusedMoE(case["e"], case["h"], case["i"], case["topk"], params_dtype=dtype, quant_config=cfg, device=DEV)
    _fill_codes(moe.w13_weight.data, gen)
    _fill_scales(moe.w13_weight_scale_inv.data, gen)
    _fill_codes(moe.w2_weight.data, gen)
    _fill_scales(moe.w2_weight_scale_inv.data, gen)
    logits = _router_logits(case, gen)
    state = {"case": case, "x": _activations(case["m"], case["h"], dtype, gen), "moe": moe}
    if case["gate"] == "softmax":
        state["logits"] = logits.to(dtype)
    else:
        state["logits"] = logits
        state["correction"] = torch.randn(case["e"], generator=gen, device=DEV).mul_(0.01)
    if case["graph"]:
        _moe(state)
        torch.cuda.synchronize()
        state["graph"] = torch.cuda.CUDAGraph()
        with torch.cuda.graph(state["graph"]):
            state["out"] = _moe(state)
    return state


# ---- one pass -------------------------------------------------------------------------------------------------------


def _moe(state):
    case = state["case"]
    if case["gate"] == "softmax":
        weights, ids = fused_topk(state["logits"], case["topk"], True)
    else:  # DeepSeek-V3's grouped routing: eight groups of experts of which four are kept
        groups = min(8, case["e"] // 4)
        weights, ids = biased_grouped_topk(state["logits"], state["correction"], case["topk"], True, groups,
                                           max(1, groups // 2), 2.5)
    return {"out": state["moe"](state["x"], StandardTopKOutput(weights, ids)), "weights": weights, "ids": ids}


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "linear":
        return state["layer"](state["x"])[0]
    if kind == "mlp":
        gate_up, _ = state["gate_up"](state["x"])
        return state["down"](ops.silu_and_mul_quant_fp8(gate_up, 128))[0]
    if kind == "quant":
        return per_token_group_quant_fp8(state["x"], 128, column_major_scales=case["column_major"],
                                         scale_tma_aligned=case["column_major"])
    if case["graph"]:
        state["graph"].replay()
        return state["out"]
    return _moe(state)


# ---- what a pass cannot do without ----------------------------------------------------------------------------------


def _weight_bytes(n, k):
    return n * k + 4 * -(-n // 128) * -(-k // 128)


def _experts_hit(case):
    """Expected number of experts that at least one of the m * topk routed rows goes to."""
    e = case["e"]
    p = [(r + 1) ** -case["skew"] for r in range(e)]
    total = sum(p)
    rows = case["m"] * case["topk"]
    return sum(1.0 - (1.0 - min(1.0, q / total)) ** rows for q in p)


def work(case):
    size = 4 if case["dtype"] == "fp32" else 2
    m, kind = case["m"], case["kind"]
    if kind == "linear":
        n, k = case["n"], case["k"]
        return {"bytes": size * m * (k + n) + _weight_bytes(n, k) + (size * n if case["bias"] else 0),
                "flops": 2 * m * n * k}
    if kind == "mlp":
        h, i = case["h"], case["i"]
        return {"bytes": 2 * size * m * h + _weight_bytes(2 * i, h) + _weight_bytes(h, i), "flops": 6 * m * h * i}
    if kind == "quant":
        k = case["k"]
        return {"bytes": m * k * (size + 1) + 4 * m * (k // 128), "flops": 0}
    h, i, rows = case["h"], case["i"], m * case["topk"]
    logit = size if case["gate"] == "softmax" else 4
    experts = _experts_hit(case) * (_weight_bytes(2 * i, h) + _weight_bytes(h, i))
    return {"bytes": 2 * size * m * h + logit * m * case["e"] + 8 * rows + int(experts), "flops": 6 * rows * h * i}


def tolerance(case):
    if case["kind"] == "quant":
        return "exact"  # codes and scales are defined bit for bit
    if case["kind"] == "linear":
        # float32 sums in another order, rounded once: half a unit in the last place of the output type
        return {"rel": 1e-3, "max": 4e-3} if case["dtype"] == "fp16" else {"rel": 4e-3, "max": 1.6e-2}
    # between the two products a 16-bit rounding may move and with it an e4m3 code of the re-quantised activations
    return {"rel": 1e-2, "max": 5e-2}
