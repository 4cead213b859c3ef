"""The one-launch route map + permute of small batches (at most 16384 routes, row-major token scales) against the oracle,
on both sides of its size limit, with masked routes and a shared expert, and with rows longer than 8192 elements."""
import numpy as np
import pytest
import torch

from helpers import compare_outputs, make_moe_case
from oracle import nvfp4_oracle as o

pytestmark = pytest.mark.gpu


def assert_layer_parity(got, ref, what):
    """The reference's acceptance rule plus a max-abs bound of 6 % of the output rms. The integer tables and the permuted
    rows are compared bit for bit above; with an intermediate size of 256 a single activation whose NVFP4 code falls on
    the other side of a rounding threshold (fast exponential on the device, exact one in the oracle) moves an output by
    up to ~5 % of the rms, so the 2 % bound of the larger layer tests does not apply to these shapes."""
    r = compare_outputs(got, ref)
    assert np.all(np.isfinite(got)), what
    assert r["mismatch"] <= 1e-3 and r["rel_l2"] <= 1e-2, (what, r)
    assert r["max_abs"] <= 6e-2 * r["rms"] + 1e-6, (what, r)


def _check_map_and_rows(p, model):
    """Integer tables, permuted payload rows and permuted scale rows of the last call, bit for bit."""
    layer = next(iter(model._layers.values()))
    ws = layer.workspace()
    ids, scores = p["topk_ids"]
    shared = int(p.get("num_fused_shared_experts") or 0)
    m = o.route_map(ids, p["num_experts"], 128, shared_experts=shared)
    etot = p["num_experts"] + shared
    t, kk = ids.shape[0], ids.shape[1] + shared
    rows = int(m["seg_start"][-1])
    assert np.array_equal(ws["counts"].cpu().numpy(), m["counts"])
    assert np.array_equal(ws["seg_start"].cpu().numpy(), m["seg_start"])
    assert np.array_equal(ws["row_of"][:t].cpu().numpy(), m["row_of"])
    n_tiles = len(m["tile_expert"])
    assert ws["totals"].cpu().numpy().tolist()[:3] == [n_tiles, rows, int((m["row_of"] >= 0).sum())]
    assert np.array_equal(ws["tile_expert"][:n_tiles].cpu().numpy(), m["tile_expert"])
    assert np.array_equal(ws["tile_rows"][:n_tiles].cpu().numpy(), m["tile_rows"])
    live = np.nonzero(m["tok_of_row"] >= 0)[0]
    tok = m["tok_of_row"][live]
    assert np.array_equal(ws["tok_of_row"][:rows].cpu().numpy()[live], tok)
    slot_w = np.concatenate([scores, np.ones((t, shared), np.float32)], axis=1) if shared else scores
    want_w = np.zeros(rows, np.float32)
    tt, ss = np.nonzero(m["row_of"] >= 0)
    want_w[m["row_of"][tt, ss]] = slot_w[tt, ss]
    assert np.array_equal(ws["weight_of_row"][:rows].cpu().numpy()[live], want_w[live])
    if not layer.cfg.tma_gather:         # otherwise FC1 gathers the token rows itself and the workspace copy is not made
        assert np.array_equal(ws["a_q"][:rows].cpu().numpy()[live], p["hidden_states"][tok])
    a_sf = o.unblock_scales(ws["a_sf"][: rows // 128].cpu().numpy().reshape(1, rows // 128, -1, 32, 16), rows,
                            p["hidden_states_scale"].shape[1])[0]
    assert np.array_equal(a_sf[live], p["hidden_states_scale"][tok])
    assert etot == len(m["counts"])


@pytest.mark.parametrize("tma_gather", [False, True])
@pytest.mark.parametrize("tokens", [1, 3, 37, 512, 1023, 1024, 1025])
def test_small_batch_map_rows_and_output(tokens, tma_gather):
    """7 routed slots + 1 shared expert = 8 routes per token, all of these sizes in one launch (16384 routes are its last).
    With the permuted copy of the payload rows and without it (FC1
    fetching the token rows by TMA gather)."""
    import kernelschema_b200 as ks
    from gpu_util import run_model
    p = make_moe_case(100 + tokens, tokens, 512, 256, 24, 7, shared=1, routing="zipf", masked=tokens > 3)
    got, _, model = run_model(p, ks.Model(tma_gather=tma_gather))
    _check_map_and_rows(p, model)
    assert_layer_parity(got, o.moe_expected(p), f"T={tokens}")


@pytest.mark.parametrize("tokens,experts,masked", [(4, 24, False), (5, 24, True), (592, 24, True), (593, 24, False), (1185, 260, True), (2047, 24, True),
                                                   (2048, 24, False), (2049, 24, True)])
def test_one_launch_map_at_the_edges_of_a_blocks_share(tokens, experts, masked):
    """8 routes per token (7 routed + 1 shared): up to 32 routes one warp of a block owns routes, from 4737 (148 blocks of 32)
    two, from 9473 four; 16384 routes are the last size of the one-launch form."""
    from gpu_util import run_model
    p = make_moe_case(400 + tokens, tokens, 256, 256, experts, 7, shared=1, routing="zipf", masked=masked)
    got, _, model = run_model(p)
    _check_map_and_rows(p, model)
    assert_layer_parity(got, o.moe_expected(p), f"T={tokens}")


def test_small_batch_hotspot_rows_stay_in_route_order():
    """Every token picks the same experts: each segment holds one row per token, in ascending token order."""
    from gpu_util import run_model
    p = make_moe_case(7, 200, 512, 256, 16, 4)
    ids = np.tile(np.array([[3, 0, 9, 15]], np.int32), (200, 1))
    p["topk_ids"] = (ids, p["topk_ids"][1])
    got, _, model = run_model(p)
    _check_map_and_rows(p, model)
    assert_layer_parity(got, o.moe_expected(p), "hotspot")


def test_small_batch_rows_longer_than_8192():
    """hidden = 8448: a row has 132 scale words, more than the 128 the first pass of the row copy moves."""
    from gpu_util import run_model
    p = make_moe_case(11, 20, 8448, 256, 4, 2)
    got, _, model = run_model(p)
    _check_map_and_rows(p, model)
    assert_layer_parity(got, o.moe_expected(p), "H=8448")


def test_repeat_calls_with_changing_batch_sizes_share_one_layer():
    """One layer object serves a large batch (2100 x 8 routes: separate route-map and permute kernels), decode batches (one launch)
    and the large batch again."""
    import kernelschema_b200 as ks
    from gpu_util import run_model
    model = ks.Model()
    for tokens in (2100, 600, 5, 2100, 64):
        p = make_moe_case(300 + tokens, tokens, 512, 256, 24, 8, routing="zipf")
        p_run = dict(p)
        got, _, model = run_model(p_run, model)
        torch.cuda.synchronize()
        assert_layer_parity(got, o.moe_expected(p), f"T={tokens}")


@pytest.mark.parametrize("tma_gather", [False, True])
@pytest.mark.parametrize("tokens", [1500, 4100])
def test_large_batch_both_payload_modes(tokens, tma_gather):
    """6000 routes (one launch) and 16400 (separate route-map and permute kernels): FC1 reading the token rows by TMA gather and FC1 reading the
    permuted copy give the same result; partially filled tiles (only some gather boxes issued) are the common case here."""
    import kernelschema_b200 as ks
    from gpu_util import run_model
    p = make_moe_case(77, tokens, 1024, 512, 16, 4, routing="zipf", masked=True)
    got, _, model = run_model(p, ks.Model(tma_gather=tma_gather))
    _check_map_and_rows(p, model)
    assert_layer_parity(got, o.moe_expected(p), f"tma_gather={tma_gather}")


@pytest.mark.parametrize("shift", [0, 1])
@pytest.mark.parametrize("tokens,top_k,hidden", [(1581, 3, 2048), (1583, 3, 2304), (3163, 3, 1024), (2047, 8, 2048)])
def test_many_routes_counted_four_at_a_time(tokens, top_k, hidden, shift):
    """Routed slots only, so the ids are counted with 128-bit loads (4743, 4749 and 9489 routes leave one or three over), and one by one
    when they do not start at a 16-byte boundary (`shift`); rows of up to 2048 elements are copied four at a time, longer ones singly."""
    import kernelschema_b200 as ks
    from gpu_util import run_model
    p = make_moe_case(500 + tokens, tokens, hidden, 256, 24, top_k, routing="zipf", masked=True)
    got, _, model = run_model(p, ks.Model(), shift_ids=shift)
    _check_map_and_rows(p, model)
    assert_layer_parity(got, o.moe_expected(p), f"T={tokens} H={hidden} shift={shift}")


@pytest.mark.parametrize("tokens,hidden,offset", [(1601, 512, 0), (1601, 512, 12), (2047, 2048, 4)])
def test_many_routes_of_which_few_are_local(tokens, hidden, offset):
    """A rank that owns four of sixteen experts, and masked routes: most of the routes that a block copies four at a time have no position.
    Tokens without a local route hold a payload of the largest code and NaN scales."""
    from gpu_util import run_model
    full = make_moe_case(700 + offset, tokens, hidden, 256, 16, 3, routing="zipf", masked=True)
    p = dict(full)
    for name in ("gemm1_weights", "gemm1_weights_scale", "gemm2_weights", "gemm2_weights_scale", "gemm1_alpha", "gemm1_beta"):
        p[name] = full[name][offset:offset + 4]
    p["num_experts"], p["local_expert_offset"] = 4, offset
    ids = full["topk_ids"][0]
    foreign = ~((ids >= offset) & (ids < offset + 4)).any(axis=1)
    assert foreign.any()
    want = o.moe_expected(p)
    p["hidden_states"], p["hidden_states_scale"] = full["hidden_states"].copy(), full["hidden_states_scale"].copy()
    p["hidden_states"][foreign], p["hidden_states_scale"].view(np.uint8)[foreign] = 0x77, 0x7F
    got, _, _ = run_model(p)
    assert_layer_parity(got, want, f"offset {offset}")
    assert not got[foreign].any()
