"""The calls whose time matters to a user of this library, with their inputs, their work and their tolerance.

A case names one public entry point (`op`), one of the synthetic model shapes of `ateniaengine_b200.synth`
(`model`) and a batch:

  layer      RealMoeLayer.forward on device activations (bf16 or f32), prefill and decode sizes
  block      RealMoeLayer.block_forward: x + MoE(rms_norm(x) * gamma), the f32 decoder-layer step
  stack      RealMoeStack.forward: a run of pre-norm residual INT8 layers, one decode step of a batch
  host       execute_real_moe_layer: the registry's operator on host f32 buffers (pinned)
  quantize   quantize_per_row_i8 of an expert matrix, or quantize_per_group_i8 and its bf16 dequant of a dense one

A layer is created with room for the largest prompt of its model and called with smaller batches too, as a
serving program does.
"""
import math

import torch

from ateniaengine_b200 import moe, synth

DEVICE = "cuda"
#: largest prompt of each shape: the capacity its layers are created with
MAX_TOKENS = {"tiny": 1024, "mixtral": 4096, "qwen_moe": 4096, "deepseek_v2_lite": 8192, "mixtral_int8": 4096}


def listed():
    return [
        # the smallest layer anyone runs (a test model's chat turn): nothing but latency and launches
        {"name": "tiny_t64", "op": "layer", "model": "tiny", "tokens": 64, "io": "f32", "v3": False},
        # one user decoding on a large bf16 model: two experts' weights per token
        {"name": "mixtral_t1", "op": "layer", "model": "mixtral", "tokens": 1, "io": "bf16", "v3": False},
        # a large decode batch or a short prompt: every expert's weights once, a few dozen rows each
        {"name": "mixtral_t256", "op": "layer", "model": "mixtral", "tokens": 256, "io": "bf16", "v3": False},
        # prefill of a long prompt, the library's headline workload
        {"name": "mixtral_t4096", "op": "layer", "model": "mixtral", "tokens": 4096, "io": "bf16", "v3": False},
        # the same through the drop-in operator of the reference: host buffers in and out
        {"name": "mixtral_host_t4096", "op": "host", "model": "mixtral", "tokens": 4096},
        # prefill on a model of many small experts with a gated shared expert
        {"name": "qwen_t2048", "op": "layer", "model": "qwen_moe", "tokens": 2048, "io": "bf16", "v3": False},
        # a short prompt of odd length through the decoder-layer step, f32 activations
        {"name": "qwen_block_t333", "op": "block", "model": "qwen_moe", "tokens": 333},
        # a decode batch of odd size on a model of many small experts
        {"name": "deepseek_t61", "op": "layer", "model": "deepseek_v2_lite", "tokens": 61, "io": "bf16", "v3": False},
        # prefill of the longest prompt on that model
        {"name": "deepseek_t8192", "op": "layer", "model": "deepseek_v2_lite", "tokens": 8192, "io": "bf16", "v3": False},
        # prefill with INT8 weights
        {"name": "mixtral_int8_t4096", "op": "layer", "model": "mixtral_int8", "tokens": 4096, "io": "bf16", "v3": False},
        # one decode step of eight users through eight INT8 layers of a large model
        {"name": "int8_stack_t8", "op": "stack", "model": "mixtral_int8", "tokens": 8, "layers": 8},
        # loading: a dense weight to INT8 in groups of 128 rows, and back to bf16 for a caller's own product
        {"name": "quantize_g128", "op": "quantize", "rows": 4096, "cols": 14336, "group": 128, "per_row": False},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    op = rng.choices(["layer", "block", "stack", "host", "quantize"], [10, 2, 2, 2, 1])[0]
    if op == "quantize":
        return {"op": op, "rows": _log_int(rng, 256, 8192), "cols": _log_int(rng, 256, 14336),
                "group": rng.choice([0, 32, 64, 128]), "per_row": rng.random() < 0.5}
    if op == "stack":
        return {"op": op, "model": "mixtral_int8", "tokens": _log_int(rng, 1, 64), "layers": rng.randint(2, 8)}
    if op == "host":
        model = rng.choice(["mixtral", "qwen_moe", "deepseek_v2_lite"])
        return {"op": op, "model": model, "tokens": _log_int(rng, 64, 4096)}
    if op == "block":
        model = rng.choice(["mixtral", "qwen_moe", "deepseek_v2_lite"])
        return {"op": op, "model": model, "tokens": _log_int(rng, 1, 2048)}
    model = rng.choice(list(MAX_TOKENS))
    return {"op": op, "model": model, "tokens": _log_int(rng, 1, MAX_TOKENS[model]),
            "io": rng.choice(["bf16", "bf16", "f32"]), "v3": model == "deepseek_v2_lite" and rng.random() < 0.25}


def _layer(shape, seed, max_tokens, v3=False):
    w = synth.make_weights(shape, seed, DEVICE)
    if not v3:
        return synth.build_layer(shape, w, max_tokens)
    # DeepSeek-V3 selection on the same layer: sigmoid scores, 8 groups of which the best 4 are kept
    gen = torch.Generator(device=DEVICE).manual_seed(seed)
    rule = {"n_group": 8, "topk_group": 4, "scaling": 2.5,
            "e_score_bias": torch.randn(shape.num_experts, generator=gen, device=DEVICE) * 0.05}
    cfg = moe.MoeLayerConfig(shape.num_experts, shape.top_k, shape.shared_d_ff > 0, shape.d_model, shape.d_ff)
    return moe.RealMoeLayer(cfg, w["router"], w["gate"], w["up"], w["down"], shared=w["shared"],
                            convention=moe.MoeExecutionConvention.Atenia, renormalize=True, max_tokens=max_tokens, v3=rule)


def prepare(case, seed):
    op = case["op"]
    if op == "quantize":
        gen = torch.Generator(device=DEVICE).manual_seed(seed)
        return {"case": case, "w": torch.randn((case["rows"], case["cols"]), generator=gen, device=DEVICE) * 0.02}
    shape, T = synth.SHAPES[case["model"]], case["tokens"]
    cap = MAX_TOKENS[case["model"]]
    f32 = op != "layer" or case["io"] == "f32"
    x = synth.make_activations(shape, seed, DEVICE, tokens=T, dtype=torch.float32 if f32 else torch.bfloat16)
    state = {"case": case, "x": x}
    if op == "stack":
        state["layers"] = [_layer(shape, 1000 * seed + l, cap) for l in range(case["layers"])]
        state["stack"] = moe.RealMoeStack(state["layers"], residual=2)
        state["out"] = torch.empty_like(x)  # a decode loop keeps its buffers
        state["stream"] = torch.cuda.Stream()
        torch.cuda.synchronize()
        return state
    state["layer"] = _layer(shape, seed, cap, case.get("v3", False))
    if op == "block":
        gen = torch.Generator(device=DEVICE).manual_seed(seed)
        state["gamma"] = 1.0 + 0.1 * torch.randn(shape.d_model, generator=gen, device=DEVICE)
    if op == "host":
        state["id"] = moe.register_resident_moe_layer(state["layer"])
        state["in"] = x.cpu().pin_memory().numpy()
        state["out"] = torch.empty(x.numel(), pin_memory=True).numpy()
    return state


def run(state):
    case = state["case"]
    op = case["op"]
    if op == "layer":
        return state["layer"].forward(state["x"])
    if op == "block":
        return state["layer"].block_forward(state["x"], gamma=state["gamma"])
    if op == "stack":
        with torch.cuda.stream(state["stream"]):
            return state["stack"].forward(state["x"], out=state["out"])
    if op == "host":
        return moe.execute_real_moe_layer(state["id"], state["in"], out=state["out"])
    if case["per_row"]:
        return moe.quantize_per_row_i8(state["w"])
    q, s = moe.quantize_per_group_i8(state["w"], case["group"])
    return q, s, moe.int8_to_bf16_per_group(q, s, case["group"])


def _touched(shape, T):
    """Experts that a batch of T tokens reaches, on average over layers drawn with the shape's routing skew."""
    gen = torch.Generator().manual_seed(0)
    L, E = 64, shape.num_experts
    logits = torch.randn(L, 512, E, generator=gen) * (0.02 * math.sqrt(shape.d_model))
    if shape.bias == "normal":
        logits += 0.5 * torch.randn(L, 1, E, generator=gen)
    elif shape.bias == "zipf":
        logits -= 1.1 * torch.log(torch.arange(1, E + 1.0))
    share = torch.zeros(L, E).scatter_add_(1, logits.topk(shape.top_k).indices.reshape(L, -1),
                                           torch.ones(L, 512 * shape.top_k)) / 512
    return float((1.0 - (1.0 - share) ** T).sum(1).mean())


def work(case):
    if case["op"] == "quantize":
        n = case["rows"] * case["cols"]
        # read f32, write the codes; the dequant reads the codes and writes bf16 (the scales are small)
        return {"bytes": n * (5 if case["per_row"] else 8), "flops": 2 * n}
    s, T = synth.SHAPES[case["model"]], case["tokens"]
    layers = case.get("layers", 1)
    weights = 3 * s.d_model * (_touched(s, T) * s.d_ff + s.shared_d_ff) * (1 if s.int8 else 2) + 4 * s.num_experts * s.d_model
    io = 2 * T * s.d_model * (2 if case["op"] == "layer" and case["io"] == "bf16" else 4)
    flops = 6 * T * s.d_model * (s.top_k * s.d_ff + s.shared_d_ff) + 2 * T * s.d_model * s.num_experts
    return {"bytes": layers * weights + io, "flops": layers * flops}


def tolerance(case):
    if case["op"] == "quantize":
        return "exact"
    # bf16 products, bf16 intermediate and expert outputs: 2.0e-3 - 2.5e-3 against the f64 oracle, times four
    return {"rel": 1e-2}
