"""Timed cases of the library's paths: the NVFP4 mixture-of-experts layer from bf16 tokens (`MoELayer.step`), the same layer
as the drop-in operator on routed NVFP4 inputs (`Model.forward`), the two dense GEMM operators (`nvfp4_quantize` +
`mm_nvfp4`, `DenseModel`) and the NVFP4 encoder alone. Sizes are those of the repository's workloads, of the operator's
fixed shapes and of the dense sweep, with odd token counts among them.

`listed()` gives the named cases, `draw(rng)` one more of the same ranges; `prepare`, `run`, `work` and `tolerance` take a case.
"""
import math

import torch

import kernelschema_b200 as ks

ACT_STD, W_STD = 1.0, 0.02
ACT_SCALE = 5.7 * ACT_STD / (6.0 * 448.0)     # calibrated global scales: block peaks of a normal sample reach about 5.7 sigma
W_SCALE = 5.7 * W_STD / (6.0 * 448.0)

# hidden, intermediate, experts, top-k, shared experts, Zipf exponent of the expert bias, largest token count
GEOMETRIES = {
    "qwen3-30b": dict(h=2048, i=768, e=128, k=8, s=0, zipf=0.0, t_max=16384),
    "qwen3-235b": dict(h=4096, i=1536, e=128, k=8, s=0, zipf=0.0, t_max=8192),
    "h4096-i768": dict(h=4096, i=768, e=128, k=8, s=0, zipf=0.0, t_max=8192),
    "deepseek-v3": dict(h=7168, i=2048, e=256, k=8, s=1, zipf=1.2, t_max=8192),
    "deepseek-v3-tp8": dict(h=7168, i=256, e=256, k=8, s=0, zipf=0.0, t_max=8192),
}


def _step(geometry, t):
    return dict(op="step", geometry=geometry, t=t)


def _forward(geometry, t, act=3, routing="balanced", clamp=False):
    return dict(op="forward", geometry=geometry, t=t, act=act, routing=routing, clamp=clamp)


def _gemm(op, m, n, k):
    return dict(op=op, m=m, n=n, k=k)


def listed():
    return [
        # one token of one interactive user through a small-expert layer: latency and launches only
        dict(_step("qwen3-30b", 1), name="decode_1_qwen3"),
        # a decode batch over the SiTU activation, almost every expert touched by a few rows
        dict(_forward("h4096-i768", 100, act=10), name="decode_100_situ"),
        # the decode batch of a large model: streams the weights of the experts that it touches
        dict(_step("deepseek-v3", 64), name="decode_64_deepseek"),
        # mixed prefill and decode, clamped activation, skewed routing: short and long expert segments side by side
        dict(_forward("qwen3-235b", 500, routing="skewed", clamp=True), name="mixed_500_clamp_skewed"),
        # one tensor-parallel slice of a large model: many experts, few rows each, a very short second reduction
        dict(_forward("deepseek-v3-tp8", 1024), name="chunk_1024_deepseek_tp8"),
        # a prefill chunk of odd length with masked routes, about one row tile per expert
        dict(_forward("qwen3-30b", 1777, routing="masked"), name="chunk_1777_qwen3_masked"),
        # prefill of many sequences, near-uniform routing
        dict(_step("qwen3-30b", 16384), name="prefill_16384_qwen3"),
        # prefill of a large model, Zipf routing and a shared expert: the headline workload
        dict(_step("deepseek-v3", 8192), name="prefill_8192_deepseek"),
        # a dense NVFP4 projection of a prefill, activations quantised on the way
        dict(_gemm("fp4", 16384, 7168, 2048), name="dense_fp4_16384"),
        # a dense projection with bf16 activations: a decode batch and a prefill
        dict(_gemm("w4a16", 16, 4096, 12288), name="dense_w4a16_16"),
        dict(_gemm("w4a16", 8192, 4096, 12288), name="dense_w4a16_8192"),
        # encoding a checkpoint matrix or a prefill's activations to NVFP4
        dict(op="encode", rows=8192, cols=7168, tiled=True, name="encode_8192x7168"),
    ]


def _log_int(rng, lo, hi):
    """Log-uniform whole number in lo..hi."""
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    op = rng.choice(["step", "step", "forward", "forward", "fp4", "w4a16", "encode"])
    if op == "step":
        g = rng.choice(["qwen3-30b", "deepseek-v3"])
        return _step(g, _log_int(rng, 1, GEOMETRIES[g]["t_max"]))
    if op == "forward":
        g = rng.choice(["qwen3-30b", "qwen3-235b", "h4096-i768", "deepseek-v3-tp8"])
        return _forward(g, _log_int(rng, 1, min(8192, GEOMETRIES[g]["t_max"])), act=rng.choice([3, 3, 10]),
                        routing=rng.choice(["balanced", "skewed", "masked", "hotspot"]), clamp=rng.random() < 0.25)
    if op == "encode":
        return dict(op="encode", rows=_log_int(rng, 64, 16384), cols=64 * _log_int(rng, 4, 128), tiled=rng.random() < 0.5)
    if op == "fp4":
        return _gemm(op, _log_int(rng, 64, 16384), 128 * _log_int(rng, 8, 64), 256 * _log_int(rng, 2, 32))
    return _gemm(op, _log_int(rng, 1, 8192), 128 * _log_int(rng, 8, 64), 256 * _log_int(rng, 4, 48))


def _generator(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed))


def _bf16(gen, shape, std):
    return torch.randn(shape, device="cuda", dtype=torch.bfloat16, generator=gen).mul_(std)


def _expert_weights(gen, experts, rows, cols):
    """NVFP4 weights [experts, rows, cols] in the operator's prepared layout (rows of a normal matrix are alike in any order)."""
    q = torch.empty((experts, rows, cols // 2), dtype=torch.uint8, device="cuda")
    sf = torch.empty((experts, rows, cols // 16), dtype=torch.uint8, device="cuda")
    step = max(1, (1 << 30) // (rows * cols))
    for j in range(0, experts, step):
        n = min(step, experts - j)
        w = _bf16(gen, (n * rows, cols), W_STD)
        ks.nvfp4_quantize(w, W_SCALE, tiled_scales=True, out=(q[j:j + n].view(n * rows, -1), sf[j:j + n].view(-1)))
    return q, sf


def _expert_bias(gen, e, zipf):
    return torch.log(1.0 / (torch.randperm(e, device="cuda", generator=gen).float() + 1.0) ** zipf)


def _prepare_step(c, gen):
    g, t = GEOMETRIES[c["geometry"]], c["t"]
    etot = g["e"] + g["s"]
    w1, s1 = _expert_weights(gen, etot, 2 * g["i"], g["h"])
    w2, s2 = _expert_weights(gen, etot, g["h"], g["i"])
    layer = ks.MoELayer(g["h"], g["i"], g["e"], g["k"], t, num_shared_experts=g["s"], graph_cache=True)
    scale_fc1 = torch.full((etot,), ACT_SCALE * W_SCALE, device="cuda")
    return dict(layer=layer, x=_bf16(gen, (t, g["h"]), ACT_STD), gate=_bf16(gen, (g["e"], g["h"]), W_STD),
                bias=_expert_bias(gen, g["e"], g["zipf"]) if g["zipf"] else None, w1=w1, s1=s1, w2=w2, s2=s2, scale_fc1=scale_fc1,
                scale_fc2=torch.full((etot,), W_SCALE, device="cuda"), out=torch.empty((t, g["h"]), dtype=torch.bfloat16, device="cuda"))


def _run_step(c, v):
    return v["layer"].step(v["x"], v["gate"], v["bias"], ACT_SCALE, v["w1"], v["s1"], v["w2"], v["s2"], v["out"],
                           scale_up=v["scale_fc1"], scale_gate=v["scale_fc1"], scale_out=v["scale_fc2"])


def _routes(c, gen):
    """Routed experts and weights as a router hands them to the operator (the operator's own routing classes)."""
    g, t = GEOMETRIES[c["geometry"]], c["t"]
    logits = torch.randn((t, g["e"]), device="cuda", generator=gen)
    if c["routing"] == "skewed":
        logits += 2.0 * torch.cos(torch.linspace(0.0, math.pi, g["e"], device="cuda"))
    if c["routing"] == "hotspot":
        logits[:, :g["k"]] += 20.0
    ids, weights = ks.route_topk(logits, g["k"])
    if c["routing"] == "masked":
        ids[::3, -1] = -1
        weights[::3, -1] = 0.0
    return ids, weights


def _prepare_forward(c, gen):
    g, t = GEOMETRIES[c["geometry"]], c["t"]
    e, h, i = g["e"], g["h"], g["i"]
    w1, s1 = _expert_weights(gen, e, 2 * i, h)
    w2, s2 = _expert_weights(gen, e, h, i)
    hq, hs = ks.nvfp4_quantize(_bf16(gen, (t, h), ACT_STD), ACT_SCALE)
    full = lambda value: torch.full((e,), value, device="cuda")
    special = c["clamp"] or c["act"] == 10          # the clamped and SiTU variants carry per-expert alpha, beta (and a limit)
    kwargs = dict(
        topk_ids=_routes(c, gen), routing_bias=None, hidden_states=hq, hidden_states_scale=hs, gemm1_weights=w1,
        gemm1_weights_scale=s1.view(torch.float8_e4m3fn), gemm1_bias=None, gemm1_alpha=full(1.702 if special else 1.0),
        gemm1_beta=full(1.0 if special else 0.0), gemm1_clamp_limit=full(7.0) if c["clamp"] else None, gemm2_weights=w2,
        gemm2_weights_scale=s2.view(torch.float8_e4m3fn), gemm2_bias=None, output1_scale_scalar=full(ACT_SCALE * W_SCALE),
        output1_scale_gate_scalar=full(ACT_SCALE * W_SCALE), output2_scale_scalar=full(W_SCALE), num_experts=e, top_k=g["k"],
        n_group=None, topk_group=None, intermediate_size=i, local_expert_offset=0, local_num_experts=e, routed_scaling_factor=1.0,
        activation_type=c["act"], output=torch.empty((t, h), dtype=torch.bfloat16, device="cuda"),
        hidden_states_scale_layout=2)
    return dict(model=ks.Model(), kwargs=kwargs)


def _run_forward(c, v):
    return v["model"](**v["kwargs"])[0]


def _prepare_fp4(c, gen):
    m, n, k = c["m"], c["n"], c["k"]
    b, b_sf = ks.nvfp4_quantize(_bf16(gen, (n, k), W_STD), W_SCALE, tiled_scales=True)
    return dict(a=_bf16(gen, (m, k), ACT_STD), b=b, b_sf=b_sf, aq=torch.empty((m, k // 2), dtype=torch.uint8, device="cuda"),
                a_sf=torch.zeros(((m + 127) // 128, k // 64, 32, 16), dtype=torch.uint8, device="cuda"),
                out=torch.empty((m, n), dtype=torch.bfloat16, device="cuda"))


def _run_fp4(c, v):
    ks.nvfp4_quantize(v["a"], ACT_SCALE, tiled_scales=True, out=(v["aq"], v["a_sf"]))
    return ks.mm_nvfp4(v["aq"], v["a_sf"], v["b"], v["b_sf"], alpha=ACT_SCALE * W_SCALE, out=v["out"])


def _prepare_w4a16(c, gen):
    m, n, k = c["m"], c["n"], c["k"]
    b, b_sf = ks.nvfp4_quantize(_bf16(gen, (n, k), W_STD), W_SCALE)
    return dict(model=ks.DenseModel(), a=_bf16(gen, (m, k), ACT_STD), b=b, b_sf=b_sf, alpha=torch.full((1,), W_SCALE, device="cuda"),
                out=torch.empty((m, n), dtype=torch.bfloat16, device="cuda"))


def _run_w4a16(c, v):
    return v["model"](v["a"], v["b"], v["b_sf"], v["alpha"], out_dtype=torch.bfloat16, out=v["out"], block_size=16)


def _prepare_encode(c, gen):
    return dict(x=_bf16(gen, (c["rows"], c["cols"]), ACT_STD))


def _run_encode(c, v):
    return ks.nvfp4_quantize(v["x"], ACT_SCALE, tiled_scales=c["tiled"])


_OPS = {
    "step": (_prepare_step, _run_step),
    "forward": (_prepare_forward, _run_forward),
    "fp4": (_prepare_fp4, _run_fp4),
    "w4a16": (_prepare_w4a16, _run_w4a16),
    "encode": (_prepare_encode, _run_encode),
}


def prepare(case, seed):
    return dict(case=case, values=_OPS[case["op"]][0](case, _generator(seed)))


def run(state):
    return _OPS[state["case"]["op"]][1](state["case"], state["values"])


def _routing_sample(c):
    """(experts touched, valid routes) of one sample of the case's routing."""
    g, t = GEOMETRIES[c["geometry"]], c["t"]
    gen = torch.Generator().manual_seed(1)
    std = math.sqrt(g["h"]) * W_STD if c["op"] == "step" else 1.0
    logits = torch.randn((t, g["e"]), generator=gen) * std
    routing = c.get("routing", "balanced")
    if g["zipf"]:
        logits += torch.log(1.0 / (torch.arange(g["e"]).float() + 1.0) ** g["zipf"])
    if routing == "skewed":
        logits += 2.0 * torch.cos(torch.linspace(0.0, math.pi, g["e"]))
    if routing == "hotspot":
        return g["k"], t * g["k"]
    ids = logits.topk(g["k"], dim=1).indices
    return int(torch.unique(ids).numel()), t * g["k"] - ((t + 2) // 3 if routing == "masked" else 0)


def work(case):
    op = case["op"]
    if op in ("step", "forward"):
        g, t = GEOMETRIES[case["geometry"]], case["t"]
        touched, routes = _routing_sample(case)
        weights = (touched + g["s"]) * 3 * g["i"] * g["h"] * 9 / 16
        tokens_in = t * g["h"] * (2 if op == "step" else 9 / 16)
        return dict(bytes=weights + tokens_in + t * g["h"] * 2 + (g["e"] * g["h"] * 2 if op == "step" else t * g["k"] * 8),
                    flops=6.0 * (routes + t * g["s"]) * g["i"] * g["h"] + (2.0 * t * g["h"] * g["e"] if op == "step" else 0.0))
    if op == "encode":
        return dict(bytes=case["rows"] * case["cols"] * (2 + 9 / 16), flops=0.0)
    m, n, k = case["m"], case["n"], case["k"]
    return dict(bytes=m * k * 2 + n * k * 9 / 16 + m * n * 2, flops=2.0 * m * n * k)


def tolerance(case):
    """About four times the distance of the path from the same arithmetic with sums, activation and weighted sum in 64 bits
    (block scales, codes and bf16 roundings as the operator defines them)."""
    op = case["op"]
    if op == "encode":
        return "exact"                              # codes and scale bytes are defined bit for bit
    if op == "step":
        return dict(rel=3e-3, max=0.5)              # a near tie of the router may send a token to another expert
    if op == "forward":
        # a last-bit difference of an FC1 sum moves an activation across a rounding threshold of E2M1 here and there (seen:
        # rel 3e-4, max 0.03); SiTU adds its hardware tanh (seen: rel 1.8e-3, max 0.06)
        return dict(rel=7e-3, max=0.25) if case["act"] == 10 else dict(rel=1.3e-3, max=0.12)
    # sums in another order flip the last bf16 bit of a few results (seen: rel 1.4e-5 and 1.5e-4, max one bf16 step)
    return dict(rel=6e-5 if op == "fp4" else 6e-4, max=1e-2)
