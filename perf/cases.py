"""The calls that the performance of this package is judged by.

A case is one pass through a public entry point as a serving program makes it: a routed-expert MoE layer
(`fused_cpp_b200.moe.fused_moe_tiled` and its routed + shared form, from given top-k arrays or from router logits), the
standalone shared MLP, or a dense W8A8 projection (`fused_cpp_b200.i8gemm`).  `listed()` names the cases that stand for
the package's real use, `draw()` gives more of the same ranges.

Layers: "v3" (H 7168, I 2048, 256 experts, top-8) and "small" (H 2048, I 1024, 16 experts, top-4) are the two
benchmark layers, "shared20" (H 4096, I 512, 20 experts + 1 shared, top-6) is the one the reference publishes times for.
Drawn cases add layers of ragged sizes.  Weights, activations, router logits and biases have the benchmark's
distributions (fused_cpp_b200/synthetic.py); router logits are N(0, 1) ("uniform") or carry a Zipf-like popularity bias
("zipf").
"""
from __future__ import annotations

import math

import torch

from fused_cpp_b200 import i8gemm, moe
from fused_cpp_b200.router import router_topk

LAYERS = {
    "v3": {"hidden": 7168, "inter": 2048, "experts": 256, "top_k": 8},
    "small": {"hidden": 2048, "inter": 1024, "experts": 16, "top_k": 4},
    "shared20": {"hidden": 4096, "inter": 512, "experts": 20, "top_k": 6},
}
# Dense projections (K, N) of the benchmark and of the attention helpers' tests.
PROJECTIONS = ((16384, 7168), (1536, 24576), (7168, 1536), (7168, 130), (2048, 272))


def _moe(path: str, layer: str, tokens: int, **options) -> dict:
    """path: w8a8 | bf16 | w8a16.  scoring: "given" (top-k arrays come from the caller) or the router's scoring."""
    case = {"op": "moe", "path": path, "tokens": tokens, "routing": "uniform", "shared": False, "activation": "silu",
            "limit": 10.0 if path == "w8a8" else 0.0, "bias": False, "scoring": "given", **LAYERS[layer]}
    case.update(options)
    return case


def _dense(rows: int, k: int, n: int, **options) -> dict:
    """n2 > 0: the paired form (two projections of the same rows)."""
    case = {"op": "dense", "rows": rows, "k": k, "n": n, "n2": 0, "input": "bf16", "output": "bf16", "bias": False}
    case.update(options)
    return case


def listed() -> list:
    return [
        # One user, one token: router logits to layer output.  The smallest call of the full-size layer.
        dict(_moe("w8a8", "v3", 1, scoring="softmax"), name="w8a8_decode_T1_router"),
        # The headline decode batch: 218 of 256 experts' weights streamed for 512 routes.
        dict(_moe("w8a8", "v3", 64), name="w8a8_decode_T64"),
        # Decode of a large batch with a prefill chunk in it, popular experts (37 hit, 1 to 500 rows each), odd size.
        dict(_moe("w8a8", "v3", 509, routing="zipf"), name="w8a8_mixed_zipf_T509"),
        # Prefill with evenly loaded experts: 256 rows each, one row more or less than a tile.
        dict(_moe("w8a8", "v3", 8192), name="w8a8_prefill_T8192"),
        # The largest call: prefill of routed experts plus the always-active shared expert.
        dict(_moe("w8a8", "v3", 16384, shared=True), name="w8a8_prefill_shared_T16384"),
        # A small model's decode step: 0.1 GB of weights, so launches and host work count.
        dict(_moe("w8a8", "small", 16), name="w8a8_small_T16"),
        # Unquantised weights, decode.
        dict(_moe("bf16", "v3", 8), name="bf16_decode_T8"),
        # The layer the reference publishes times for, at the largest of its three batch sizes.
        dict(_moe("bf16", "shared20", 2048, shared=True, limit=10.0), name="bf16_shared20_T2048"),
        # Unquantised prefill, popular experts, odd size.
        dict(_moe("bf16", "v3", 4095, routing="zipf"), name="bf16_prefill_zipf_T4095"),
        # A checkpoint with interleaved gate/up rows, the swigluoai activation and biases, mid-size batch.
        dict(_moe("bf16", "small", 200, activation="swigluoai", bias=True), name="bf16_swigluoai_bias_T200"),
        # int8 weights with 16-bit activations, a prefill chunk of ragged size.
        dict(_moe("w8a16", "v3", 1000), name="w8a16_T1000"),
        # Dense W8A8 attention output projection of a decode batch.
        dict(_dense(64, 16384, 7168), name="dense_decode_64"),
    ]


def _spread(rng, low: int, high: int) -> int:
    """Log-uniform over [low, high]; any residue."""
    return max(low, min(high, round(math.exp(rng.uniform(math.log(low), math.log(high + 1))))))


def _seconds(case: dict) -> float:
    """Rough time of a pass, to keep drawn cases below the largest listed one."""
    w = work(case)
    rate = 2.0e15 if case.get("path") == "w8a8" or case["op"] == "dense" else 1.0e15
    return max(w["bytes"] / 6.0e12, w["flops"] / rate)


def _draw_moe(rng) -> dict:
    path = rng.choice(("w8a8", "w8a8", "w8a8", "bf16", "bf16", "w8a16"))
    layer = rng.choice(("v3", "v3", "small", "shared20", "ragged"))
    sizes = dict(LAYERS.get(layer, {}))
    if not sizes:
        experts = rng.randint(2, 96)
        sizes = {"hidden": 16 * rng.randint(16, 320), "inter": 16 * rng.randint(8, 160), "experts": experts,
                 "top_k": rng.randint(1, min(9, experts))}
    case = _moe(path, "v3", _spread(rng, 1, 16384), routing=rng.choice(("uniform", "uniform", "zipf")),
                shared=rng.random() < 0.25, **sizes)
    if not case["shared"]:
        if path != "w8a8":  # (the planner runtime that W8A16 goes through takes SiLU only)
            kind = rng.choice(("silu", "silu", "clamp", "gelu", "swigluoai") if path == "bf16" and layer != "v3" else ("silu", "clamp"))
            case["activation"] = "silu" if kind == "clamp" else kind
            case["limit"] = 10.0 if kind == "clamp" else 0.0
        case["bias"] = path == "bf16" and rng.random() < 0.3
        case["scoring"] = rng.choice(("given", "given", "softmax", "sigmoid"))
    return case


def draw(rng) -> dict:
    kind = rng.random()
    if kind < 0.70:
        case = _draw_moe(rng)
    elif kind < 0.95:
        k, n = rng.choice(PROJECTIONS + ((rng.randint(64, 8192), rng.randint(64, 8192)),))
        case = _dense(_spread(rng, 1, 8192), k, n)
        if rng.random() < 0.3:
            case["n2"] = rng.choice((1536, 8192, 520))
        else:
            case.update(input=rng.choice(("bf16", "bf16", "f32")), output=rng.choice(("bf16", "bf16", "f32")), bias=rng.random() < 0.3)
    else:
        hidden, inter = rng.choice(((7168, 2048), (4096, 512), (2048, 1024)))
        case = {"op": "mlp", "rows": _spread(rng, 1, 8192), "hidden": hidden, "inter": inter, "limit": rng.choice((0.0, 10.0))}
    bound = 0.8 * _seconds(_moe("w8a8", "v3", 16384, shared=True))
    size = "tokens" if case["op"] == "moe" else "rows"
    while _seconds(case) > bound:
        case[size] = case[size] * 2 // 3 + 1
    return case


# ---- inputs --------------------------------------------------------------------------------------------------------

def _routing_logits(case: dict, generator: torch.Generator) -> torch.Tensor:
    device = generator.device
    logits = torch.randn((case["tokens"], case["experts"]), generator=generator, device=device)
    if case["routing"] == "zipf":
        rank = torch.randperm(case["experts"], generator=generator, device=device).to(torch.float32)
        logits += 2.0 * torch.log(1.0 / (rank + 1.0))
    return logits


def _int8_weight(shape: tuple, generator: torch.Generator):
    weight = torch.empty(shape, dtype=torch.int8, device=generator.device).random_(-127, 128, generator=generator)
    scale = torch.empty(shape[:-1], device=generator.device).uniform_(0.5, 2.0, generator=generator)
    return weight, scale.div_(127.0 * math.sqrt(shape[-1]))


def _bf16_weight(shape: tuple, generator: torch.Generator) -> torch.Tensor:
    return torch.empty(shape, dtype=torch.bfloat16, device=generator.device).normal_(0.0, 0.02, generator=generator)


def _activations(rows: int, columns: int, generator: torch.Generator) -> torch.Tensor:
    return torch.empty((rows, columns), dtype=torch.bfloat16, device=generator.device).normal_(0.0, 1.0, generator=generator)


def _moe_weights(case: dict, generator: torch.Generator):
    """The prepared weights; the routed + shared form holds the shared expert as expert id E."""
    hidden, inter = case["hidden"], case["inter"]
    experts = case["experts"] + (1 if case["shared"] else 0)
    if case["path"] == "bf16":
        packed = moe.prepare_fused_moe_bf16_tiled_weights(_bf16_weight((experts, 2 * inter, hidden), generator),
                                                          _bf16_weight((experts, hidden, inter), generator), fuse_silu=True)
        holder = moe.PreparedBF16TiledRoutedSharedMoEWeights
    else:
        w13, s13 = _int8_weight((experts, 2 * inter, hidden), generator)
        w2, s2 = _int8_weight((experts, hidden, inter), generator)
        if case["path"] == "w8a8":
            packed = moe.prepare_fused_moe_w8a8_tiled_quantized_weights(w13, s13, w2, s2)
            holder = moe.PreparedW8A8TiledRoutedSharedMoEWeights
        else:
            packed = moe.prepare_fused_moe_w8a16_tiled_quantized_weights(w13, s13, w2, s2)
            holder = moe.PreparedW8A16TiledRoutedSharedMoEWeights
    return holder(packed, case["experts"], case["experts"]) if case["shared"] else packed


def _prepare_moe(case: dict, generator: torch.Generator) -> dict:
    state = {"weights": _moe_weights(case, generator), "x": _activations(case["tokens"], case["hidden"], generator)}
    logits = _routing_logits(case, generator)
    if case["scoring"] == "given":
        values, ids = torch.topk(torch.softmax(logits, dim=-1), case["top_k"], dim=-1)
        state["topk_weights"] = (values / values.sum(dim=-1, keepdim=True)).contiguous()
        state["topk_ids"] = ids.contiguous()
    else:
        state["logits"] = logits
        if case["scoring"] == "sigmoid":
            state["selection_bias"] = 0.1 * torch.randn(case["experts"], generator=generator, device=generator.device)
    if case["bias"]:
        for name, channels in (("w13_bias", 2 * case["inter"]), ("w2_bias", case["hidden"])):
            state[name] = _bf16_weight((case["experts"], channels), generator)
    # The planner runtime a serving program installs once: the library's automatic tiles.
    runtime = moe.MoePlannerRuntime(None, hidden_size=case["hidden"], intermediate_size=case["inter"], global_experts=case["experts"],
                                    local_experts=case["experts"], shared_experts=1 if case["shared"] else 0)
    moe.set_default_moe_planner_runtime(runtime)
    return state


def prepare(case: dict, seed: int) -> dict:
    generator = torch.Generator(device="cuda").manual_seed(seed)
    state = {"case": case}
    if case["op"] == "moe":
        state.update(_prepare_moe(case, generator))
    elif case["op"] == "mlp":
        state["x"] = _activations(case["rows"], case["hidden"], generator)
        state["weights"] = moe.prepare_shared_mlp_bf16_tiled_weights(_bf16_weight((2 * case["inter"], case["hidden"]), generator),
                                                                     _bf16_weight((case["hidden"], case["inter"]), generator))
    else:
        x = _activations(case["rows"], case["k"], generator)
        state["x"] = x.float() if case["input"] == "f32" else x
        state["weight"] = i8gemm.prepare(*_int8_weight((case["n"], case["k"]), generator))
        if case["n2"]:
            state["second"] = i8gemm.prepare(*_int8_weight((case["n2"], case["k"]), generator))
        state["bias"] = _activations(1, case["n"], generator)[0] if case["bias"] else None
    return state


# ---- one pass ------------------------------------------------------------------------------------------------------

def _run_moe(case: dict, state: dict):
    if case["shared"]:
        forward = {"w8a8": moe.fused_moe_w8a8_tiled_with_shared, "bf16": moe.fused_moe_bf16_tiled_with_shared,
                   "w8a16": moe.fused_moe_w8a16_tiled_with_shared}[case["path"]]
        return forward(state["x"], state["weights"], state["topk_weights"], state["topk_ids"], swiglu_limit=case["limit"])
    routed = None
    if case["scoring"] != "given":
        routed = router_topk(state["logits"], case["top_k"], scoring=case["scoring"], selection_bias=state.get("selection_bias"))
    weights, ids = routed or (state["topk_weights"], state["topk_ids"])
    out = moe.fused_moe_tiled(state["x"], state["weights"], weights, ids, w13_bias=state.get("w13_bias"), w2_bias=state.get("w2_bias"),
                              activation=case["activation"], swiglu_limit=case["limit"])
    return {"out": out, "topk_weights": weights, "topk_ids": ids} if routed else out


def run(state: dict):
    case = state["case"]
    if case["op"] == "moe":
        return _run_moe(case, state)
    if case["op"] == "mlp":
        return moe.shared_mlp_bf16_tiled(state["x"], state["weights"], swiglu_limit=case["limit"])
    if case["n2"]:
        return i8gemm.dynamic_scaled_mm_pair(state["x"], state["weight"], state["second"])
    out_dtype = torch.float32 if case["output"] == "f32" else torch.bfloat16
    return i8gemm.dynamic_scaled_mm(state["x"], state["weight"], bias=state["bias"], out_dtype=out_dtype)


# ---- what a pass cannot do without ---------------------------------------------------------------------------------

def _experts_hit(case: dict) -> int:
    """Experts that a routing of the case's distribution reaches (one fixed sample)."""
    logits = _routing_logits(case, torch.Generator().manual_seed(1))
    return int(torch.unique(torch.topk(logits, case["top_k"], dim=-1).indices).numel())


def work(case: dict) -> dict:
    """Bytes: the weights of the experts that are hit, the inputs and the outputs, once each.  Flops: the products' (for
    int8 operands: integer operations)."""
    if case["op"] == "dense":
        rows, k, n = case["rows"], case["k"], case["n"] + case["n2"]
        moved = rows * k * (4 if case["input"] == "f32" else 2) + n * (k + 4) + rows * n * (4 if case["output"] == "f32" else 2)
        return {"bytes": moved, "flops": 2 * rows * k * n}
    hidden, inter = case["hidden"], case["inter"]
    if case["op"] == "mlp":
        return {"bytes": 6 * hidden * inter + 4 * case["rows"] * hidden, "flops": 6 * case["rows"] * hidden * inter}
    tokens, top_k = case["tokens"], case["top_k"]
    channels = 2 * inter + hidden
    per_expert = 6 * hidden * inter if case["path"] == "bf16" else 3 * hidden * inter + 4 * channels
    per_expert += 2 * channels if case["bias"] else 0
    moved = (_experts_hit(case) + (1 if case["shared"] else 0)) * per_expert + 4 * tokens * hidden + 12 * tokens * top_k
    moved += 0 if case["scoring"] == "given" else 4 * tokens * case["experts"]
    routes = tokens * (top_k + (1 if case["shared"] else 0))
    return {"bytes": moved, "flops": 6 * routes * hidden * inter}


def tolerance(case: dict):
    """int8 operands: integer sums and a fixed sequence of fp32 roundings, so the outputs are defined bit for bit (the
    reference's order of operations).  With the router in front, an ulp of its fp32 softmax flips single bf16 roundings
    of the output: with 64-bit routing weights the output moves by 1.3e-5 relative (2-norm), single values by 0.7e-2.
    bf16 operands: the order of the fp32 sums is free, which flips bf16 roundings of the intermediate and of the output;
    against 64-bit sums the output moves by 0.6e-3 (2.5e-3 with an unrounded intermediate), single values by 1.4e-2."""
    if case["op"] == "dense" or (case["op"] == "moe" and case["path"] != "bf16" and case["scoring"] == "given"):
        return "exact"
    if case["op"] == "moe" and case["path"] != "bf16":
        return {"rel": 6e-5, "max": 2.8e-2}
    return {"rel": 5e-3, "max": 3e-2}
