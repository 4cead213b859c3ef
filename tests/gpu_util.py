"""GPU-side test plumbing: numpy case -> torch CUDA tensors -> the library's Model, with guard bands."""
import numpy as np
import torch

import kernelschema_b200 as ks


def to_dev(a, dtype=None):
    if a is None:
        return None
    t = torch.from_numpy(np.ascontiguousarray(a)).cuda()
    return t if dtype is None else t.view(dtype)


def guarded_output(t, h):
    """Output view inside a larger allocation filled with -17, as the reference generator makes it (input.py:48-51)."""
    backing = torch.full((t * h + 128,), -17, dtype=torch.bfloat16, device="cuda")
    return backing, backing[64:-64].view(t, h)


def run_model(p, model=None, shift_ids=0):
    """Run the drop-in Model on a numpy case; returns (output fp32 numpy, backing tensor, model). `shift_ids`: the expert ids start that
    many elements behind a 256-byte boundary."""
    model = model or ks.Model()
    ids, scores = p["topk_ids"]
    t = p["hidden_states"].shape[0]
    h = p["hidden_states"].shape[1] * 2
    backing, out = guarded_output(t, h)
    etot = p["gemm1_weights"].shape[0]
    shared = int(p.get("num_fused_shared_experts") or 0)
    ids_dev = to_dev(ids.astype(np.int32))
    if shift_ids:
        ids_dev = torch.cat([ids_dev.new_zeros(shift_ids), ids_dev.flatten()])[shift_ids:].view(ids_dev.shape)
    kw = dict(
        topk_ids=(ids_dev, to_dev(scores.astype(np.float32))), routing_bias=None,
        hidden_states=to_dev(p["hidden_states"]), hidden_states_scale=to_dev(p["hidden_states_scale"], torch.float8_e4m3fn),
        gemm1_weights=to_dev(p["gemm1_weights"]), gemm1_weights_scale=to_dev(p["gemm1_weights_scale"], torch.float8_e4m3fn),
        gemm1_bias=None, gemm1_alpha=to_dev(p["gemm1_alpha"]), gemm1_beta=to_dev(p["gemm1_beta"]),
        gemm1_clamp_limit=to_dev(p.get("gemm1_clamp_limit")), gemm2_weights=to_dev(p["gemm2_weights"]),
        gemm2_weights_scale=to_dev(p["gemm2_weights_scale"], torch.float8_e4m3fn), gemm2_bias=None,
        output1_scale_scalar=to_dev(p.get("output1_scale_scalar", np.ones(etot, np.float32))),
        output1_scale_gate_scalar=to_dev(p.get("output1_scale_gate_scalar", np.ones(etot, np.float32))),
        output2_scale_scalar=to_dev(p.get("output2_scale_scalar", np.ones(etot, np.float32))),
        num_experts=int(p["num_experts"]), top_k=int(p["top_k"]), n_group=None, topk_group=None,
        intermediate_size=int(p["intermediate_size"]), local_expert_offset=int(p.get("local_expert_offset") or 0),
        local_num_experts=etot - shared, routed_scaling_factor=1.0, routing_method_type=0, do_finalize=True, enable_pdl=False,
        activation_type=int(p.get("activation_type", 3)), per_token_scale=None, output=out, tune_max_num_tokens=max(t, 1),
        gemm1_lora_delta=None, valid_hidden_size=None, valid_intermediate_size=None,
        num_fused_shared_experts=shared or None, hidden_states_scale_layout=2)
    snapshot = {k: v.clone() for k, v in kw.items() if isinstance(v, torch.Tensor) and k != "output"}
    res = model(**kw)
    torch.cuda.synchronize()
    assert isinstance(res, list) and res[0] is out, "forward must return [output] (same tensor object)"
    for k, v in snapshot.items():
        assert torch.equal(v.view(torch.uint8), kw[k].view(torch.uint8)), f"input {k} was modified"
    guard = torch.cat([backing[:64], backing[-64:]]).float()
    assert bool((guard == -17).all()), "bytes outside the output view were written"
    for layer in model._layers.values():
        assert layer.status() == 0, "a bounded device wait expired"
    return out.float().cpu().numpy(), kw, model
