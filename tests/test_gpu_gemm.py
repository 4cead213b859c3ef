"""GPU parity of the tcgen05 NVFP4 GEMM (dense entry point) against the oracle's dequantise-then-matmul."""
import ctypes as C

import numpy as np
import pytest
import torch

from conftest import load_golden
from helpers import compare_outputs
from oracle import nvfp4_oracle as o

pytestmark = pytest.mark.gpu


def _dense_case(m, n, k, seed, tile_n, alpha=1.0, a_scale=1.0):
    import kernelschema_b200 as ks
    rng = np.random.default_rng(seed)
    a = o.bf16_round(rng.standard_normal((m, k), dtype=np.float32) * a_scale)
    b = o.bf16_round(rng.standard_normal((n, k), dtype=np.float32) * 0.02)
    bq, bs = o.quantize(b)
    a_dev = torch.from_numpy(o.bf16_bits(a).view(np.int16)).cuda().view(torch.bfloat16)
    aq, asf = ks.nvfp4_quantize(a_dev, 1.0, tiled_scales=True)
    status = torch.zeros(4, dtype=torch.int32, device="cuda")
    bsf_t = ks.scales_to_tiles(torch.from_numpy(bs).cuda())
    out = ks.mm_nvfp4(aq, asf, torch.from_numpy(bq).cuda(), bsf_t, alpha=alpha, tile_n=tile_n, status=status)
    torch.cuda.synchronize()
    assert int(status[0]) == 0, f"bounded device wait expired: code {int(status[0])}"
    oq, os_ = o.quantize(a)
    assert np.array_equal(aq.cpu().numpy(), oq)
    ref = o.dense_expected(o.decode(oq, os_), bq, bs, alpha)
    return out.float().cpu().numpy(), ref


@pytest.mark.parametrize("m,n,k,tile_n", [(128, 128, 256, 128), (128, 256, 256, 256), (192, 256, 512, 128),
                                          (192, 256, 512, 256), (1000, 1024, 2048, 128), (1000, 1024, 2048, 256),
                                          (5, 128, 7168, 128), (2048, 2048, 2048, 256), (256, 256, 256, 512),
                                          (192, 256, 512, 512), (1000, 1024, 2048, 512), (5, 256, 7168, 512),
                                          (2048, 2048, 2048, 512), (4096 + 128, 512, 1024, 512)])
def test_dense_gemm_matches_oracle(m, n, k, tile_n):
    got, ref = _dense_case(m, n, k, seed=m + n + k, tile_n=tile_n, alpha=0.75)
    r = compare_outputs(got, ref)
    # exact products, fp32 accumulation in a different order: at most a bf16 ulp on a few elements
    assert r["rel_l2"] <= 2e-3, r
    ulp_off = (o.bf16_bits(got) != o.bf16_bits(ref)).mean()
    assert ulp_off <= 0.05, ulp_off
    assert r["max_abs"] <= 2e-2 * r["rms"], r


@pytest.mark.parametrize("m,n,k,tile_n", [(128 * 600, 128, 256, 128), (128 * 400, 256, 512, 256), (256 * 300, 256, 512, 512),
                                          (128 * 330, 512, 768, 256)])
def test_dense_gemm_many_items_per_cta(m, n, k, tile_n):
    """Short K and several work items per CTA (or CTA pair): the stage ring and the per-stage scale-factor buffers wrap
    across tiles, the accumulator phases flip and the tile-table entries are prefetched one item ahead."""
    got, ref = _dense_case(m, n, k, seed=7 + tile_n, tile_n=tile_n)
    r = compare_outputs(got, ref)
    assert r["rel_l2"] <= 2e-3 and r["max_abs"] <= 2e-2 * r["rms"], r
    assert (o.bf16_bits(got) != o.bf16_bits(ref)).mean() <= 0.05


def test_dense_gemm_golden_weights():
    """B operand and scales from the reference's dense problem generator; A quantised on the device."""
    import kernelschema_b200 as ks
    g = load_golden("dense")
    a = o.bf16_from_bits(g["a"])
    aq, asf = ks.nvfp4_quantize(torch.from_numpy(g["a"].view(np.int16)).cuda().view(torch.bfloat16), 1.0, tiled_scales=True)
    out = ks.mm_nvfp4(aq, asf, torch.from_numpy(g["b"]).cuda(), ks.scales_to_tiles(torch.from_numpy(g["b_descale"]).cuda()),
                      alpha=float(g["alpha"][0]))
    oq, os_ = o.quantize(a)
    ref = o.dense_expected(o.decode(oq, os_), g["b"], g["b_descale"], float(g["alpha"][0]))
    r = compare_outputs(out.float().cpu().numpy(), ref)
    assert r["rel_l2"] <= 2e-3 and r["max_abs"] <= 2e-2 * r["rms"], r
    # against the reference's own output (bf16 A, not quantised): only the A quantisation error remains
    r2 = compare_outputs(out.float().cpu().numpy(), o.bf16_from_bits(g["out"]))
    assert r2["rel_l2"] <= 0.12, r2


def test_dense_gemm_linearity_full_size():
    """Size-independent property at a benchmark size: scaling A by 2 (exact in bf16 and in the block scales) doubles the output."""
    import kernelschema_b200 as ks
    gen = torch.Generator(device="cuda").manual_seed(3)
    a = torch.randn(4096, 4096, device="cuda", generator=gen).to(torch.bfloat16)
    b = (torch.randn(4096, 4096, device="cuda", generator=gen) * 0.02).to(torch.bfloat16)
    bq, bsf = ks.nvfp4_quantize(b, 1.0, tiled_scales=True)
    outs = []
    for s in (1.0, 2.0):
        aq, asf = ks.nvfp4_quantize((a * s).to(torch.bfloat16), 1.0, tiled_scales=True)
        outs.append(ks.mm_nvfp4(aq, asf, bq, bsf, tile_n=256).float())
    assert torch.equal(outs[0] * 2, outs[1])
    # spot-check 64 rows against the oracle
    rows = torch.arange(0, 4096, 64)
    aq, asf = ks.nvfp4_quantize(a, 1.0)
    bq_r, bs_r = ks.nvfp4_quantize(b, 1.0)
    ref = o.dense_expected(o.decode(aq[rows].cpu().numpy(), asf.view(torch.uint8)[rows].cpu().numpy()), bq_r.cpu().numpy(),
                           bs_r.view(torch.uint8).cpu().numpy())
    r = compare_outputs(outs[0][rows].cpu().numpy(), ref)
    assert r["rel_l2"] <= 2e-3 and r["max_abs"] <= 2e-2 * r["rms"], r


# ----------------------------------------------------------------------------- bf16 x NVFP4 (A not quantised)
def _w4a16_case(m, n, k, seed, outliers=False):
    rng = np.random.default_rng(seed)
    a = o.bf16_round(rng.standard_normal((m, k), dtype=np.float32) * np.linspace(0.65, 1.35, k, dtype=np.float32))
    if outliers:
        a[:, ::64] = o.bf16_round(a[:, ::64] * 8.0)
    w = o.bf16_round(rng.standard_normal((n, k), dtype=np.float32) * np.float32(k ** -0.5))
    bq, bsf = o.quantize(w)
    return a, bq, bsf


def _bf16_dev(a):
    return torch.from_numpy(o.bf16_bits(a).view(np.int16)).cuda().view(torch.bfloat16)


def test_w4a16_matches_reference_output_bits():
    """The reference's own dense problem (bf16 A, its generator's B, scales and alpha) and its own output: the weights
    are expanded exactly, so only the order of the fp32 additions differs (a bf16 ulp on a few elements)."""
    import kernelschema_b200 as ks
    g = load_golden("dense")
    a = torch.from_numpy(g["a"].view(np.int16)).cuda().view(torch.bfloat16)
    backing = torch.full((192 * 256 + 128,), -17, dtype=torch.bfloat16, device="cuda")
    out = backing[64:-64].view(192, 256)
    inputs = [a.clone(), torch.from_numpy(g["b"]).cuda(), torch.from_numpy(g["b_descale"]).cuda(), torch.from_numpy(g["alpha"]).cuda()]
    snap = [t.clone() for t in inputs]
    status = torch.zeros(1, dtype=torch.int32, device="cuda")
    res = ks.DenseModel()(inputs[0], inputs[1], inputs[2].view(torch.float8_e4m3fn), inputs[3], backend="blackwell-native",
                          out_dtype=torch.bfloat16, out=out, block_size=16, enable_pdl=False)
    torch.cuda.synchronize()
    assert res is out and int(status.item()) == 0
    assert all(torch.equal(x, y) for x, y in zip(inputs, snap))                  # inputs preserved
    assert (backing[:64] == -17).all() and (backing[-64:] == -17).all()          # nothing written outside `out`
    got, ref = out.float().cpu().numpy(), o.bf16_from_bits(g["out"])
    r = compare_outputs(got, ref)
    assert r["rel_l2"] <= 1e-3 and r["max_abs"] <= 2e-2 * r["rms"], r
    # the reference's own acceptance rule (metadata.json: atol 0.01, rtol 0.05, no mismatch allowed)
    assert (np.abs(got - ref) <= 0.01 + 0.05 * np.abs(ref)).all()
    assert (o.bf16_bits(got) != o.bf16_bits(ref)).mean() <= 0.05


@pytest.mark.parametrize("m,n,k,outliers", [(1, 128, 256, False), (100, 256, 512, False), (129, 384, 768, True), (256, 128, 2048, False),
                                            (300, 1536, 1024, False), (1000, 512, 256, True), (300, 384, 512, False),
                                            (513, 768, 1024, False)])
def test_w4a16_matches_oracle(m, n, k, outliers):
    import kernelschema_b200 as ks
    a, bq, bsf = _w4a16_case(m, n, k, 100 + m, outliers)
    alpha = torch.tensor([0.75], dtype=torch.float32, device="cuda")
    status = torch.zeros(1, dtype=torch.int32, device="cuda")
    out = ks.mm_bf16_nvfp4(_bf16_dev(a), torch.from_numpy(bq).cuda(), torch.from_numpy(bsf).cuda(), alpha, status=status)
    torch.cuda.synchronize()
    assert int(status.item()) == 0
    ref = o.dense_expected(a, bq, bsf, 0.75)
    got = out.float().cpu().numpy()
    r = compare_outputs(got, ref)
    assert r["rel_l2"] <= 1e-3 and r["max_abs"] <= 2e-2 * r["rms"], r
    assert (np.abs(got - ref) <= 0.01 + 0.05 * np.abs(ref)).all()
    assert (o.bf16_bits(got) != o.bf16_bits(ref)).mean() <= 0.05


@pytest.mark.parametrize("m,n,k", [(1, 128, 256), (7, 384, 2304), (8, 4096, 12288), (9, 1024, 4096), (16, 8192, 512), (17, 256, 2048),
                                   (31, 7168, 768), (32, 128, 12288), (17, 8192, 4096),
                                   (32, 8192, 4352), (20, 1024, 12288), (24, 9600, 2048)])
def test_w4a16_decode_sizes_all_codes(m, n, k):
    """A handful of tokens, and from 17 rows on both sides of the rule that leaves long K (32 x 8192 x 4352) and a second wave of
    blocks (24 x 9600 x 2048) to the tile kernel: every code and every scale byte (subnormal scales and the 0.5 code among them)
    in random places, a strided A, and rows beyond M left alone. Sums of K products differ from the oracle's only by the order of the fp32
    additions, so a bf16 step (2^-8) of the result plus 2^-20 of the sum of magnitudes bounds every element."""
    import kernelschema_b200 as ks
    rng = np.random.default_rng(m + n + k)
    wide = torch.zeros((m, k + 8), dtype=torch.bfloat16, device="cuda")
    a = o.bf16_round(rng.standard_normal((m, k), dtype=np.float32))
    wide[:, :k] = _bf16_dev(a)
    bq = rng.integers(0, 256, (n, k // 2), dtype=np.uint8)
    bsf = rng.integers(0, 0x7F, (n, k // 16), dtype=np.uint8)
    backing = torch.full((m + 2, n), -17.0, dtype=torch.bfloat16, device="cuda")
    out = ks.mm_bf16_nvfp4(wide[:, :k], torch.from_numpy(bq).cuda(), torch.from_numpy(bsf).cuda(),
                           torch.tensor([0.5], dtype=torch.float32, device="cuda"), out=backing[1:m + 1])
    torch.cuda.synchronize()
    assert (backing[0] == -17).all() and (backing[m + 1] == -17).all()
    codes = np.array([0, 0.5, 1, 1.5, 2, 3, 4, 6, -0.0, -0.5, -1, -1.5, -2, -3, -4, -6], dtype=np.float64)
    w = np.empty((n, k))
    w[:, 0::2], w[:, 1::2] = codes[bq & 15], codes[bq >> 4]
    scale = torch.arange(256, dtype=torch.int32).to(torch.uint8).view(torch.float8_e4m3fn).double().numpy()[bsf]
    w *= np.repeat(scale, 16, axis=1)
    ref, mag = 0.5 * a.astype(np.float64) @ w.T, 0.5 * np.abs(a).astype(np.float64) @ np.abs(w).T
    assert (np.abs(out.float().cpu().numpy() - ref) <= np.abs(ref) / 256 + mag * 2.0 ** -20).all()


def test_w4a16_strided_a_and_no_alpha():
    import kernelschema_b200 as ks
    a, bq, bsf = _w4a16_case(64, 128, 512, 7)
    wide = torch.zeros((64, 512 + 64), dtype=torch.bfloat16, device="cuda")
    wide[:, :512] = _bf16_dev(a)
    out = ks.mm_bf16_nvfp4(wide[:, :512], torch.from_numpy(bq).cuda(), torch.from_numpy(bsf).cuda())
    ref = o.dense_expected(a, bq, bsf, 1.0)
    r = compare_outputs(out.float().cpu().numpy(), ref)
    assert r["rel_l2"] <= 1e-3, r


@pytest.mark.parametrize("m,n,k", [(2047, 2048, 4096), (2048, 2048, 4096), (2049, 1024, 4352), (2048, 2048, 3840)])
def test_dense_both_sides_of_the_long_loop_form(m, n, k):
    """K >= 4096 and M >= 2048 copies the scale factors in line with eight epilogue warps, other launches use copier warps:
    the same bits as 128-wide tiles on both sides of each limit (same products, same order along K)."""
    import kernelschema_b200 as ks
    gen = torch.Generator(device="cuda").manual_seed(m + k)
    aq, asf = ks.nvfp4_quantize(torch.randn(m, k, device="cuda", generator=gen).to(torch.bfloat16), tiled_scales=True)
    bq, bsf = ks.nvfp4_quantize(torch.randn(n, k, device="cuda", generator=gen).to(torch.bfloat16), tiled_scales=True)
    wide = ks.mm_nvfp4(aq, asf, bq, bsf, tile_n=256)
    narrow = ks.mm_nvfp4(aq, asf, bq, bsf, tile_n=128)
    torch.cuda.synchronize()
    assert torch.equal(wide, narrow) and wide.float().abs().mean() > 1


@pytest.mark.parametrize("m,n,k", [(33, 4096, 8192), (128, 4096, 8192), (129, 256, 256), (300, 1024, 1280), (513, 4096, 4096), (2600, 4096, 4096),
                                   (3000, 3328, 4352), (77, 20480, 4096), (40, 640, 2304), (128, 45056, 8192)])
def test_w4a16_split_last_wave(m, n, k):
    """Up to 128 rows: problems of fewer tiles than SMs, and a last wave behind whole ones (20480 columns: 160 tiles, 12 of them split
    on 148 SMs; 45056: 176 wide tiles, 28 split). More rows: never split. The same sums with and without the workspace up to the
    order of the fp32 additions, rows beyond M left alone."""
    import kernelschema_b200 as ks
    gen = torch.Generator(device="cuda").manual_seed(m + n)
    a = torch.randn(m, k, device="cuda", generator=gen).to(torch.bfloat16)
    bq, bsf = ks.nvfp4_quantize((torch.randn(n, k, device="cuda", generator=gen) * k ** -0.5).to(torch.bfloat16), 1.0)
    alpha = torch.tensor([1.25], dtype=torch.float32, device="cuda")
    backing = torch.full((m + 2, n), -17.0, dtype=torch.bfloat16, device="cuda")
    y = ks.mm_bf16_nvfp4(a, bq, bsf.view(torch.uint8), alpha, out=backing[1:m + 1])
    plain = ks.mm_bf16_nvfp4(a, bq, bsf.view(torch.uint8), alpha, split_k=False)
    torch.cuda.synchronize()
    assert (backing[0] == -17).all() and (backing[m + 1] == -17).all()
    codes = torch.tensor([0, .5, 1, 1.5, 2, 3, 4, 6, 0, -.5, -1, -1.5, -2, -3, -4, -6], device="cuda", dtype=torch.float64)
    w = torch.stack((codes[(bq & 15).long()], codes[(bq >> 4).long()]), -1).view(n, k)
    w = (w.view(n, k // 16, 16) * bsf.view(torch.float8_e4m3fn).double()[..., None]).view(n, k)
    ref, mag = 1.25 * a.double() @ w.T, 1.25 * a.double().abs() @ w.abs().T
    for got in (y, plain):          # one bf16 rounding, and 2^-20 of the magnitudes for the fp32 sums
        assert ((got.double() - ref).abs() <= ref.abs() / 256 + mag * 2.0 ** -20).all()


def test_w4a16_split_on_two_streams_and_in_a_graph():
    """Calls on different streams keep apart (each stream its own scratch), and a captured call still gives its result after
    larger calls have replaced the stream's scratch."""
    import kernelschema_b200 as ks
    gen = torch.Generator(device="cuda").manual_seed(9)
    m, n, k = 60, 2048, 4096
    a = [torch.randn(m, k, device="cuda", generator=gen).to(torch.bfloat16) for _ in range(2)]
    bq, bsf = ks.nvfp4_quantize((torch.randn(n, k, device="cuda", generator=gen) * k ** -0.5).to(torch.bfloat16), 1.0)
    bsf = bsf.view(torch.uint8)
    want = [ks.mm_bf16_nvfp4(x, bq, bsf) for x in a]
    torch.cuda.synchronize()
    streams = [torch.cuda.Stream() for _ in range(2)]
    outs = [[torch.empty_like(want[0]) for _ in range(20)] for _ in range(2)]
    for r in range(20):
        for i, st in enumerate(streams):
            with torch.cuda.stream(st):
                ks.mm_bf16_nvfp4(a[i], bq, bsf, out=outs[i][r])
    torch.cuda.synchronize()
    assert all(torch.equal(outs[i][r], want[i]) for i in range(2) for r in range(20))
    out = torch.empty_like(want[0])
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        ks.mm_bf16_nvfp4(a[0], bq, bsf, out=out)
    ks.mm_bf16_nvfp4(torch.cat((a[0], a[1])), bq, bsf)
    graph.replay()
    torch.cuda.synchronize()
    assert torch.equal(out, want[0])


@pytest.mark.parametrize("n,k,sizes", [(4096, 4096, (129, 300, 1024, 1025, 1280, 1281, 2600)), (3328, 4352, (200, 3000)), (1152, 8192, (150, 1300)),
                                       (4096, 8192, (33, 64, 65, 128)), (20480, 4096, (40, 128)), (4096, 12288, (1, 8, 9, 16)), (2048, 7168, (17, 24, 32)),
                                       (6144, 8192, (17, 24, 32)), (1024, 12288, (17, 32))])
def test_w4a16_a_row_has_one_value(n, k, sizes):
    """A row gives the same bits at any position and in any batch of 1..16, 17..32, 33..128 and more than 128 rows: long K, fewer
    tiles than SMs (128-wide up to 1024 rows x 4096, 256-wide above) as well as a partly filled last wave behind whole ones. With split_k=False the bits are those of more than 128
    rows at every size."""
    import kernelschema_b200 as ks
    gen = torch.Generator(device="cuda").manual_seed(n + k)
    m = sizes[-1]
    a = torch.randn(m, k, device="cuda", generator=gen).to(torch.bfloat16)
    bq, bsf = ks.nvfp4_quantize((torch.randn(n, k, device="cuda", generator=gen) * k ** -0.5).to(torch.bfloat16), 1.0)
    bsf = bsf.view(torch.uint8)
    y = ks.mm_bf16_nvfp4(a, bq, bsf)
    perm = torch.randperm(m, device="cuda", generator=gen)
    assert torch.equal(ks.mm_bf16_nvfp4(a[perm].contiguous(), bq, bsf), y[perm])
    for t in sizes:
        assert torch.equal(ks.mm_bf16_nvfp4(a[m - t:], bq, bsf), y[m - t:]), t
    # without a split the three ranges agree as well
    plain = ks.mm_bf16_nvfp4(a.repeat(200 // m + 1, 1)[:max(m, 200)], bq, bsf)
    for t in (1, 8, 16, 17, 32, 33, 128, *sizes):
        if t <= m:
            assert torch.equal(ks.mm_bf16_nvfp4(a[:t], bq, bsf, split_k=False), plain[:t]), t


def test_w4a16_linearity_full_size():
    """Size-independent properties at a reference shape (M 8192, N 4096, K 2048): doubling A doubles the output exactly,
    and a row of A gives the same output row whatever tile it sits in."""
    import kernelschema_b200 as ks
    gen = torch.Generator(device="cuda").manual_seed(5)
    a = torch.randn(8192, 2048, device="cuda", generator=gen).to(torch.bfloat16)
    w = (torch.randn(4096, 2048, device="cuda", generator=gen) * 2048 ** -0.5).to(torch.bfloat16)
    bq, bsf = ks.nvfp4_quantize(w, 1.0)
    y1 = ks.mm_bf16_nvfp4(a, bq, bsf.view(torch.uint8))
    y2 = ks.mm_bf16_nvfp4((a * 2).to(torch.bfloat16), bq, bsf.view(torch.uint8))
    assert torch.equal(y1.float() * 2, y2.float())
    perm = torch.randperm(8192, device="cuda", generator=gen)
    y3 = ks.mm_bf16_nvfp4(a[perm].contiguous(), bq, bsf.view(torch.uint8))
    assert torch.equal(y3, y1[perm])
    assert y1.float().abs().mean() > 0.1


def test_w4a16_rejects_bad_shapes():
    import kernelschema_b200 as ks
    a = torch.zeros((8, 128), dtype=torch.bfloat16, device="cuda")
    with pytest.raises((ValueError, RuntimeError)):
        ks.mm_bf16_nvfp4(a, torch.zeros((128, 64), dtype=torch.uint8, device="cuda"), torch.zeros((128, 8), dtype=torch.uint8, device="cuda"))


@pytest.mark.parametrize("m,n,k", [(16, 4096, 3072), (128, 1024, 2048), (1, 256, 1024), (100, 7168, 2048)])
def test_w4a16_split_k_small_m(m, n, k):
    """Small M: several CTAs share one output tile through fp32 partial sums added in a fixed order. Same result as the
    one-CTA-per-tile form up to the order of the fp32 additions, and identical from run to run."""
    import kernelschema_b200 as ks
    a, bq, bsf = _w4a16_case(m, n, k, 300 + m)
    args = (_bf16_dev(a), torch.from_numpy(bq).cuda(), torch.from_numpy(bsf).cuda(), torch.tensor([1.25], dtype=torch.float32, device="cuda"))
    y_split = ks.mm_bf16_nvfp4(*args, split_k=True)
    y_again = ks.mm_bf16_nvfp4(*args, split_k=True)
    y_plain = ks.mm_bf16_nvfp4(*args, split_k=False)
    torch.cuda.synchronize()
    assert torch.equal(y_split, y_again)
    ref = o.dense_expected(a, bq, bsf, 1.25)
    for y in (y_split, y_plain):
        got = y.float().cpu().numpy()
        r = compare_outputs(got, ref)
        assert r["rel_l2"] <= 1e-3 and r["max_abs"] <= 2e-2 * r["rms"], r
        assert (np.abs(got - ref) <= 0.01 + 0.05 * np.abs(ref)).all()


@pytest.mark.parametrize("m,n,k", [(129, 128, 1280), (256, 384, 2304), (257, 1152, 4096), (300, 640, 1280), (385, 4096, 12288), (1025, 2176, 1536),
                                   (3000, 1280, 2304)])
def test_w4a16_expanded_weights(m, n, k):
    """Above 128 rows the weights are expanded to bf16 first: every payload byte and every finite scale code, odd rows (a last row tile of
    1, 44 and 129 rows), a half-empty 256-wide column tile, both tile widths, expansions of one and of several waves, ten calls in a
    row. Same bits as the kernel that decodes tile by tile; that one and the product agree with 64-bit sums to half a bf16 step (at most
    2^-8 of the element, whose significand has eight bits) plus fp32 accumulation (k * 2^-24 of the sum of magnitudes at most)."""
    import kernelschema_b200 as ks
    from kernelschema_b200 import _lib
    assert _lib.load().b200moe_gemm_bf16_nvfp4_workspace_bytes(m, n, k) == n * k * 2
    gen = torch.Generator(device="cuda").manual_seed(m + n)
    wide = torch.randn(m, k + 8, device="cuda", generator=gen).to(torch.bfloat16)
    a = wide[:, :k]
    bq = torch.randint(0, 256, (n, k // 2), dtype=torch.uint8, device="cuda", generator=gen)
    sf = torch.randint(0, 127, (n, k // 16), dtype=torch.uint8, device="cuda", generator=gen)
    sf |= torch.randint(0, 2, sf.shape, dtype=torch.uint8, device="cuda", generator=gen) << 7
    alpha = torch.full((1,), 2.0 ** -9, device="cuda")
    y = [ks.mm_bf16_nvfp4(a, bq, sf, alpha) for _ in range(10)]
    want = ks.mm_bf16_nvfp4(a, bq, sf, alpha, split_k=False)
    assert all(torch.equal(v, want) for v in y)
    code = torch.tensor([0, 0.5, 1, 1.5, 2, 3, 4, 6, -0.0, -0.5, -1, -1.5, -2, -3, -4, -6], device="cuda", dtype=torch.float64)
    w = code[torch.stack([bq & 15, bq >> 4], dim=-1).long()].view(n, k) * sf.view(torch.float8_e4m3fn).double().repeat_interleave(16, dim=1)
    rows = torch.unique(torch.cat([torch.arange(min(m, 130)), torch.arange(m - 130, m)])).cuda()
    x = a[rows].double()
    exact, mag = (x @ w.t()) * 2.0 ** -9, (x.abs() @ w.abs().t()) * 2.0 ** -9
    assert ((y[0][rows].double() - exact).abs() <= exact.abs() * 2.0 ** -8 + mag * (k * 2.0 ** -24)).all()


@pytest.mark.parametrize("offset", [0, 16, 32, 48])
def test_w4a16_workspace_of_a_c_caller(offset):
    """Above 128 rows the C entry takes a workspace on any 16-byte boundary. On a 32-byte boundary the weights are expanded into its
    n * k * 2 bytes and nothing behind them is written; on a 16-byte boundary only it is left alone. Same bits."""
    import kernelschema_b200 as ks
    from kernelschema_b200 import _lib
    m, n, k = 200, 1152, 4096
    lib = _lib.load()
    need = lib.b200moe_gemm_bf16_nvfp4_workspace_bytes(m, n, k)
    assert need == n * k * 2
    gen = torch.Generator(device="cuda").manual_seed(offset)
    a = torch.randn(m, k, device="cuda", generator=gen).to(torch.bfloat16)
    bq = torch.randint(0, 256, (n, k // 2), dtype=torch.uint8, device="cuda", generator=gen)
    sf = torch.randint(0, 127, (n, k // 16), dtype=torch.uint8, device="cuda", generator=gen)
    want = ks.mm_bf16_nvfp4(a, bq, sf, split_k=False)
    ws = torch.full((need + 64,), 0xA5, dtype=torch.uint8, device="cuda")
    assert ws.data_ptr() % 64 == 0
    out = torch.empty_like(want)
    stream = torch.cuda.current_stream().cuda_stream
    rc = lib.b200moe_gemm_bf16_nvfp4(a.data_ptr(), k, bq.data_ptr(), sf.data_ptr(), None, out.data_ptr(), m, n, k, n,
                                     ws.data_ptr() + offset, need, None, stream)
    assert rc == 0 and torch.equal(out, want)
    written = ws != 0xA5
    assert not written[:offset].any() and not written[offset + need:].any()
    assert written.any() == (offset % 32 == 0)


def _weights(gen, n, k):
    import kernelschema_b200 as ks
    q, s = ks.nvfp4_quantize((torch.randn(n, k, device="cuda", generator=gen) * k ** -0.5).to(torch.bfloat16), 1.0)
    return q, s.view(torch.uint8)


def test_w4a16_many_rows_on_two_streams_and_in_a_graph(monkeypatch):
    """Above 128 rows: calls on two streams keep apart while each takes and returns its scratch; a captured call still gives its result
    after the memory around it has been used by others; without scratch the result is the same."""
    import kernelschema_b200 as ks
    from kernelschema_b200 import ops
    gen = torch.Generator(device="cuda").manual_seed(9)
    m, n, k = 300, 2048, 4096
    a = [torch.randn(m, k, device="cuda", generator=gen).to(torch.bfloat16) for _ in range(2)]
    w = [_weights(gen, n, k) for _ in range(2)]
    want = [ks.mm_bf16_nvfp4(a[i], *w[i], split_k=False) for i in range(2)]
    streams = [torch.cuda.Stream() for _ in range(2)]
    outs = [[torch.empty_like(want[0]) for _ in range(20)] for _ in range(2)]
    torch.cuda.synchronize()
    for r in range(20):
        for i, st in enumerate(streams):
            with torch.cuda.stream(st):
                ks.mm_bf16_nvfp4(a[i], *w[i], out=outs[i][r])
    torch.cuda.synchronize()
    assert all(torch.equal(outs[i][r], want[i]) for i in range(2) for r in range(20))

    out = [torch.empty_like(v) for v in want]
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        held = ops._w4a16_expanded(a[0].device, 4096)
        assert held is not None                     # in a graph of torch's the expanded weights have a place
        for i in range(2):
            ks.mm_bf16_nvfp4(a[i], *w[i], out=out[i])
    others = [torch.full((n * k * 2,), 0x5A, dtype=torch.uint8, device="cuda") for _ in range(4)]
    for _ in range(3):
        out[0].zero_(), out[1].zero_()
        ks.mm_bf16_nvfp4(torch.cat(a), *w[0])
        graph.replay()
        torch.cuda.synchronize()
        assert torch.equal(out[0], want[0]) and torch.equal(out[1], want[1])
    assert all((v == 0x5A).all() for v in others)

    monkeypatch.setattr(ops, "_w4a16_expanded", lambda device, need: None)
    assert torch.equal(ks.mm_bf16_nvfp4(a[0], *w[0]), want[0])


@pytest.mark.parametrize("m", [60, 300])
def test_w4a16_in_a_capture_that_torch_did_not_begin(m):
    """The allocator has no pool for such a graph, so the call must not keep scratch of the allocator's in it: what is allocated after the
    capture stays as it is when the graph is replayed, and the outputs are those of a call without scratch."""
    import kernelschema_b200 as ks
    rt = C.CDLL("libcudart.so.12")                  # torch's, loaded already
    gen = torch.Generator(device="cuda").manual_seed(m)
    n, k = 2048, 4096
    a, w = torch.randn(m, k, device="cuda", generator=gen).to(torch.bfloat16), _weights(gen, n, k)
    want = ks.mm_bf16_nvfp4(a, *w, split_k=m <= 128)
    out, st = torch.zeros_like(want), torch.cuda.Stream()
    torch.cuda.synchronize()
    with torch.cuda.stream(st):
        graph, exe = C.c_void_p(), C.c_void_p()
        assert rt.cudaStreamBeginCapture(C.c_void_p(st.cuda_stream), 0) == 0
        try:
            ks.mm_bf16_nvfp4(a, *w, out=out)
        finally:
            rc = rt.cudaStreamEndCapture(C.c_void_p(st.cuda_stream), C.byref(graph))
        assert rc == 0 and rt.cudaGraphInstantiateWithFlags(C.byref(exe), graph, C.c_ulonglong(0)) == 0
        others = [torch.full((n * k * 2,), 0x5A, dtype=torch.uint8, device="cuda") for _ in range(4)]
        for _ in range(3):
            assert rt.cudaGraphLaunch(exe, C.c_void_p(st.cuda_stream)) == 0
        st.synchronize()
        assert all((v == 0x5A).all() for v in others)
    scale = want.float().pow(2).mean().sqrt()       # up to 128 rows the sums run in another order without scratch
    assert torch.equal(out, want) if m > 128 else (out.float() - want.float()).abs().max() <= scale * 2.0 ** -5
    assert rt.cudaGraphExecDestroy(exe) == 0 and rt.cudaGraphDestroy(graph) == 0


def test_cluster_kernels_between_launches_of_several_waves():
    """Quantiser launches of several waves of blocks before and behind every kernel that runs as clusters, ten rounds without a
    synchronize in between: the outputs of the calls one by one."""
    import kernelschema_b200 as ks
    gen = torch.Generator(device="cuda").manual_seed(1)
    x = torch.randn((8192, 4096), device="cuda", generator=gen).to(torch.bfloat16)
    w, w_sf = ks.nvfp4_quantize(x[:4096], 1.0)
    w_sft, w_sf = ks.scales_to_tiles(w_sf), w_sf.view(torch.uint8)
    calls = (lambda: ks.nvfp4_quantize(x, 0.5)[0], lambda: ks.mm_bf16_nvfp4(x[:16], w, w_sf), lambda: ks.nvfp4_quantize(x, 0.25)[0],
             lambda: ks.router_logits(x[:256], x[:128]), lambda: ks.nvfp4_quantize(x, 0.125)[0],
             lambda: ks.mm_nvfp4(w[:512], w_sft[:4], w, w_sft, tile_n=512), lambda: ks.mm_bf16_nvfp4(x[:129], w, w_sf))
    want = []
    for call in calls:
        want.append(call())
        torch.cuda.synchronize()
    got = [[call() for call in calls] for _ in range(10)]
    torch.cuda.synchronize()
    assert all(torch.equal(g, v) for row in got for g, v in zip(row, want))


@pytest.mark.parametrize("m,n,k", [(1, 256, 512), (130, 512, 2304), (128, 18944, 512), (128, 19200, 512), (4736, 512, 768), (4737, 512, 768)])
def test_dense_gemm_default_tile_width(m, n, k):
    """tile_n = 0 on both sides of the line where the 128-wide tiles stop running at once (148 of them): the bits of either explicit width."""
    import kernelschema_b200 as ks
    gen = torch.Generator(device="cuda").manual_seed(m + n)
    aq, asf = ks.nvfp4_quantize(torch.randn(m, k, device="cuda", generator=gen).to(torch.bfloat16), 1.0, tiled_scales=True)
    bq, bsf = ks.nvfp4_quantize(torch.randn(n, k, device="cuda", generator=gen).to(torch.bfloat16), 1.0, tiled_scales=True)
    y = [ks.mm_nvfp4(aq, asf, bq, bsf, alpha=0.5, tile_n=t) for t in (0, 128, 256)]
    assert torch.equal(y[0], y[1]) and torch.equal(y[0], y[2])
