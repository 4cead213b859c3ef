// Dense GEMM with bf16 activations and NVFP4 weights (W4A16): out = bf16(alpha * A @ decode(B)^T), the contract of
// gemm/dense/bf16_nvfp4_gemm/problem/reference.py:10-15 (A is NOT quantised; B payload [N, K/2] with row-major,
// un-swizzled E4M3 block-16 scales [N, K/16]).
//
// An E2M1 value times an E4M3 scale has at most 6 significant bits and lies in [2^-10, 2688], so it is exactly
// representable in bf16. The weights are therefore expanded to bf16 on the fly, bit-exactly, and the
// product runs on tcgen05.mma kind::f16 (bf16 x bf16, fp32 accumulation in TMEM): the result differs from the fp32
// reference only by the order of the fp32 additions.
//
// Tile: 256 rows of A (two 128-row accumulators) x BN weight rows, K in steps of 64; one decoded weight tile feeds two
// MMAs. Weight loads, decoding, operand traffic and MMAs share an SM's time and none alone is the bound (8192 x 4096 x 12288,
// 734 us, with one part left out: no weight loads 554, no MMAs 596, no decoding 614). The wide form BN = 256 is taken where N and
// the number of tiles allow it (w4a16_plan) because it moves less for the same work: 160 KB of shared-memory traffic per
// 256 x 256 x 64 step against 112 KB per 256 x 128 x 64 step. Its two 256-column accumulators fill the 512 TMEM columns, so the
// epilogue of a tile (a few microseconds) is not overlapped; BN = 128 alternates between two accumulator pairs.
// Warp roles: 0 = TMA producer of A (bf16, 128-byte swizzle); 1 = TMEM owner + MMA issuer; then BN/32 decoder warps, one
// thread per weight row of the tile. In the wide form a warp loads its 32 rows' lines (128 bytes = 256 weights each) one k-group
// ahead, four rows per instruction, and turns them to a row per lane in a shared-memory patch of its own: loaded row by row, an
// instruction touches 32 lines, and those passes through the L1 pipe compete with the operand traffic (8192 x 4096 x 12288
// 796 us, 759 through the patch). A thread expands its row with byte permutes and one bf16 multiply per pair, and writes bf16 into
// shared memory in the layout a 128-byte-swizzled TMA load would have produced (16-byte chunk c of row r at
// r * 128 + ((c ^ (r & 7)) * 16)), then fence.proxy.async + mbarrier arrive; the last 8 warps = epilogue.
// Every wait is bounded and reports through the status word.
//
// Above 128 rows this kernel serves calls without a workspace and the few shapes where expanding the weights first is not faster
// (gemm_w4a16_expand.cu, the same bits).
//
// Up to 128 rows the tiles of a last, partly filled wave are split along K (fp32 partial tiles, added in split order by
// k_w4a16_reduce) as long as that fills the idle SMs; a problem with fewer tiles than SMs is all tail. From 129 rows on nothing is
// split: every element is one sum in ascending k, whatever tile and batch its row sits in.
#include "kernels.cuh"
#include "ptx.cuh"
#include "w4a16.cuh"

namespace b200 {

namespace {

template <int BN>
struct WCfg {
  static constexpr int kStages = BN == 256 ? 3 : 4;
  static constexpr int kABytes = 256 * 128;                // 256 rows x 64 bf16
  static constexpr int kBBytes = BN * 128;                 // BN weight rows x 64 bf16
  static constexpr int kDecWarps = BN / 32;                // one decoder thread per weight row
  static constexpr bool kPatch = BN == 256;                // weights through a patch: the narrow form has few, short tiles to
                                                           // hide the extra trip behind (M = 128, N = 2048, K = 4096: 13.8 -> 15.7 us)
  static constexpr int kPatchBytes = kPatch ? 32 * 128 : 0;   // per decoder warp
  static constexpr int kSmem = kStages * (kABytes + kBBytes) + kDecWarps * kPatchBytes + 1024 + 256;
  static constexpr int kEpiWarp0 = 2 + kDecWarps;          // first epilogue warp: 2 mod 4, so warp & 3 walks the lane quadrants
  static constexpr int kThreads = 32 * (kEpiWarp0 + 8);
  static constexpr int kAccBufs = 256 / BN;                // pairs of accumulators that fit the 512 TMEM columns
};

struct W4A16Params {
  const uint8_t* b_q;      // [N, K/2]
  const uint8_t* b_sf;     // [N, K/16] E4M3, row-major
  const float* alpha;      // device scalar or null (= 1)
  __nv_bfloat16* out;
  int64_t out_stride;
  int M, N, K;
  int32_t* status;
  // Tiles from `full_tiles` on are shared by `splits` CTAs, each of which reduces `groups_per_split` k-groups of 256 and writes
  // fp32 sums to partial[split][tile - full_tiles][M][BN] (M <= 128: one row tile). splits == 1: no workspace, full_tiles = all.
  int full_tiles, tail_tiles;
  int splits;
  int groups_per_split;
  float* partial;
};

DEV void fence_async_proxy() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }

// Half of one k-step (32 of its 64 weights) of one weight row: four payload words and their two scale bytes (low 16
// bits of sf2) -> 64 bytes of bf16. `dst` is the row's base inside the stage; 16-byte chunk c (= c0 + 0..3) goes to
// chunk slot c ^ sw (the 128-byte swizzle, sw = row & 7). Magnitude x scale is exact in bf16 (2 x 4 significant bits).
DEV void decode_half_stage(const uint32_t* w, uint32_t sf2, uint32_t dst, uint32_t sw, uint32_t c0) {
  const uint32_t sc_pair = e4m3x2_to_bf16x2(sf2);
#pragma unroll
  for (int j = 0; j < 4; ++j) {                     // 16-byte chunk = 8 weights = one payload word; two chunks share a scale
    const uint32_t c = c0 + j;
    const uint32_t sc = (j & 2) ? __byte_perm(sc_pair, 0, 0x3232) : __byte_perm(sc_pair, 0, 0x1010);
    uint32_t o[4];
    e2m1x4_to_bf16x2(w[j], o[0], o[1]);
    e2m1x4_to_bf16x2(w[j] >> 16, o[2], o[3]);
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const __nv_bfloat162 prod = __hmul2(*reinterpret_cast<const __nv_bfloat162*>(&o[i]), *reinterpret_cast<const __nv_bfloat162*>(&sc));
      o[i] = *reinterpret_cast<const uint32_t*>(&prod);
    }
    asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(dst + ((c ^ sw) << 4)), "r"(o[0]), "r"(o[1]), "r"(o[2]), "r"(o[3])
                 : "memory");
  }
}

// BN accumulator columns of the calling warp's 32 lanes -> alpha * x as bf16 at out[row, col0 ...], 64 columns at a
// time, or as fp32 at `partial_row`; `release` is called right after the last TMEM read. A warp without live rows only releases.
template <int BN, class Release>
DEV void store_cols(const W4A16Params& p, uint32_t taddr, int row, bool live, int col0, float alpha, float* partial_row, Release release) {
  if (!__any_sync(0xFFFFFFFFu, live)) {
    release();
    return;
  }
  if (partial_row) {                                 // alpha and the rounding come in the reduce
#pragma unroll
    for (int pass = 0; pass < BN / 32; ++pass) {
      float v[32];
      tmem_ld32(taddr + pass * 32, v);
      tmem_ld_wait();
      if (pass == BN / 32 - 1) release();
      if (live) {
#pragma unroll
        for (int j = 0; j < 8; ++j)
          reinterpret_cast<float4*>(partial_row + pass * 32)[j] = make_float4(v[4 * j], v[4 * j + 1], v[4 * j + 2], v[4 * j + 3]);
      }
    }
    return;
  }
  __nv_bfloat16* dst_row = p.out + (size_t)row * p.out_stride + col0;
#pragma unroll
  for (int pass = 0; pass < BN / 64; ++pass) {
    float v[2][32];
    tmem_ld32(taddr + pass * 64, v[0]);
    tmem_ld32(taddr + pass * 64 + 32, v[1]);
    tmem_ld_wait();
    if (pass == BN / 64 - 1) release();
    if (live) {
#pragma unroll
      for (int cb = 0; cb < 2; ++cb) {
        uint32_t o[16];
#pragma unroll
        for (int j = 0; j < 16; ++j) {
          const __nv_bfloat162 pr = __floats2bfloat162_rn(v[cb][2 * j] * alpha, v[cb][2 * j + 1] * alpha);
          o[j] = *reinterpret_cast<const uint32_t*>(&pr);
        }
        __nv_bfloat16* d = dst_row + pass * 64 + cb * 32;
#pragma unroll
        for (int j = 0; j < 2; ++j)
          asm volatile("st.global.L1::no_allocate.v8.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};" ::"l"(d + 16 * j), "r"(o[8 * j]),
                       "r"(o[8 * j + 1]), "r"(o[8 * j + 2]), "r"(o[8 * j + 3]), "r"(o[8 * j + 4]), "r"(o[8 * j + 5]), "r"(o[8 * j + 6]),
                       "r"(o[8 * j + 7])
                       : "memory");
      }
    }
  }
}

template <int BN>
__global__ void __launch_bounds__(WCfg<BN>::kThreads, 1)
k_gemm_w4a16(const __grid_constant__ CUtensorMap tm_a, const W4A16Params p) {
  using C = WCfg<BN>;
  extern __shared__ uint8_t smem_raw[];
  const uint32_t base = (smem_u32(smem_raw) + 1023u) & ~1023u;
  const uint32_t s_a = base, s_b = s_a + C::kStages * C::kABytes, s_patch = s_b + C::kStages * C::kBBytes;
  const uint32_t s_bar = s_patch + C::kDecWarps * C::kPatchBytes;
  const uint32_t bar_full_a = s_bar;                         // [stages] TMA bytes of A landed
  const uint32_t bar_full_b = bar_full_a + 8 * C::kStages;   // [stages] the decoder warps wrote their rows
  const uint32_t bar_empty = bar_full_b + 8 * C::kStages;    // [stages] MMAs of the stage retired
  const uint32_t bar_acc_full = bar_empty + 8 * C::kStages;  // [kAccBufs]
  const uint32_t bar_acc_empty = bar_acc_full + 16;          // [kAccBufs] 8 epilogue warps
  const uint32_t s_slot = bar_acc_empty + 16;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;

  if (threadIdx.x == 0) {
    for (int s = 0; s < C::kStages; ++s) {
      mbar_init(bar_full_a + 8 * s, 1);
      mbar_init(bar_full_b + 8 * s, C::kDecWarps);
      mbar_init(bar_empty + 8 * s, 1);
    }
    for (int b = 0; b < C::kAccBufs; ++b) {
      mbar_init(bar_acc_full + 8 * b, 1);
      mbar_init(bar_acc_empty + 8 * b, 8);
    }
    mbar_init_fence();
    tma_prefetch_desc(&tm_a);
  }
  if (warp == 1) tmem_alloc<512>(s_slot);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  uint32_t tmem;
  asm volatile("ld.shared.u32 %0, [%1];" : "=r"(tmem) : "r"(s_slot));
  pdl_wait();

  const int n_nt = p.N / BN;                // BN-row tiles of the weights
  const int groups = p.K >> 8;              // k-groups of 256 weights = one 128-byte line per weight row
  // items: the whole tiles, then (tail tile, split) with the split fastest; tile = (mt, nt), n fastest: the CTAs of a wave share
  // A's rows and sweep the weights (L2-resident). A split covers k-groups [g0, g1).
  const int total_items = p.full_tiles + p.tail_tiles * p.splits;
  struct Item {
    int tile, split, g0, g1;                // split -1: the whole of K
  };
  auto item_at = [&](int item) -> Item {    // once per item and role: the divisions cost a few hundred cycles
    const int t = item - p.full_tiles;
    if (t < 0) return {item, -1, 0, groups};
    const int q = t / p.splits, s = t - q * p.splits;
    return {p.full_tiles + q, s, s * p.groups_per_split, min(groups, (s + 1) * p.groups_per_split)};
  };

  if (warp == 0) {
    // ------------------------------------------------------------------ TMA producer of A
    if (lane == 0) {
      uint32_t s = 0, ph = 1;
      bool ok = true;
      for (int item = blockIdx.x; ok && item < total_items; item += gridDim.x) {
        const Item at = item_at(item);
        const int mt = at.tile / n_nt, ks1 = 4 * at.g1;
        for (int ks = 4 * at.g0; ks < ks1; ++ks) {
          if (!mbar_wait(bar_empty + 8 * s, ph)) { if (p.status) atomicCAS(p.status, 0, 121); ok = false; break; }
          mbar_expect_tx(bar_full_a + 8 * s, C::kABytes);
          tma_load_2d(s_a + s * C::kABytes, &tm_a, bar_full_a + 8 * s, ks * 128, mt * 256);
          if (++s == C::kStages) { s = 0; ph ^= 1; }
        }
      }
      pdl_trigger();
    }
  } else if (warp == 1) {
    // ------------------------------------------------------------------ MMA issuer
    if (lane == 0) {
      constexpr uint32_t idesc = make_idesc_bf16(128, BN);
      uint32_t s = 0, ph = 0, it = 0;
      bool ok = true;
      for (int item = blockIdx.x; ok && item < total_items; item += gridDim.x, ++it) {
        const Item at = item_at(item);
        const bool second = p.M - at.tile / n_nt * 256 > 128;          // rows 128..255 of the tile hold real rows
        const int nk = 4 * (at.g1 - at.g0);
        const uint32_t buf = it % C::kAccBufs;
        if (!mbar_wait(bar_acc_empty + 8 * buf, ((it / C::kAccBufs) & 1) ^ 1)) { if (p.status) atomicCAS(p.status, 0, 122); break; }
        tc_fence_after();
        const uint32_t acc = tmem + buf * 2 * BN;
        for (int ks = 0; ks < nk; ++ks) {
          if (!mbar_wait(bar_full_a + 8 * s, ph) || !mbar_wait(bar_full_b + 8 * s, ph)) {
            if (p.status) atomicCAS(p.status, 0, 123);
            ok = false;
            break;
          }
          tc_fence_after();
          const uint64_t a_d = make_desc_sw128(s_a + s * C::kABytes), b_d = make_desc_sw128(s_b + s * C::kBBytes);
#pragma unroll
          for (int q = 0; q < 4; ++q) {
            mma_bf16(acc, a_d + 2 * q, b_d + 2 * q, idesc, (ks | q) ? 1u : 0u);
            if (second) mma_bf16(acc + BN, a_d + (128 * 128 >> 4) + 2 * q, b_d + 2 * q, idesc, (ks | q) ? 1u : 0u);
          }
          mma_commit(bar_empty + 8 * s);
          if (++s == C::kStages) { s = 0; ph ^= 1; }
        }
        if (ok) mma_commit(bar_acc_full + 8 * buf);
      }
    }
  } else if (warp < C::kEpiWarp0) {
    // ------------------------------------------------------------------ weight decoders: thread = weight row of the tile
    const int r = threadIdx.x - 64;                         // 0 .. BN-1
    const uint32_t row_off = (uint32_t)r * 128u;
    const uint32_t sw = (uint32_t)(r & 7);
    uint32_t s = 0, ph = 1;
    bool ok = true;
    uint4 nxt[8];
    uint4 nxt_sf;
    const uint32_t patch = s_patch + (uint32_t)(warp - 2) * C::kPatchBytes;
    // one k-group of the warp's rows: through the patch lane -> row 4i + lane / 8, 16-byte piece lane % 8, else each lane its own
    // row; and the scales of the lane's own row
    auto fetch = [&](const Item& at, int g) {
      const size_t row0 = (size_t)(at.tile % n_nt) * BN + (r & ~31);
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        const int row = C::kPatch ? 4 * i + (lane >> 3) : lane, piece = C::kPatch ? lane & 7 : i;
        nxt[i] = __ldg(reinterpret_cast<const uint4*>(p.b_q + (row0 + row) * (size_t)(p.K >> 1)) + (size_t)g * 8 + piece);
      }
      nxt_sf = __ldg(reinterpret_cast<const uint4*>(p.b_sf + (row0 + lane) * (size_t)(p.K >> 4)) + g);
    };
    Item at = item_at(blockIdx.x);
    if ((int)blockIdx.x < total_items) fetch(at, at.g0);
    for (int item = blockIdx.x; ok && item < total_items; item += gridDim.x) {
      const Item cur_item = at;
      const int g1 = at.g1;
      if (item + (int)gridDim.x < total_items) at = item_at(item + gridDim.x);      // the next item
      for (int g = cur_item.g0; ok && g < g1; ++g) {
        uint32_t line[C::kPatch ? 1 : 32];
        if constexpr (!C::kPatch) {
#pragma unroll
          for (int i = 0; i < 8; ++i) {
            line[4 * i] = nxt[i].x; line[4 * i + 1] = nxt[i].y; line[4 * i + 2] = nxt[i].z; line[4 * i + 3] = nxt[i].w;
          }
        }
        if (C::kPatch) __syncwarp();                        // the previous group has been read out of the patch
#pragma unroll
        for (int i = 0; C::kPatch && i < 8; ++i) {
          const uint32_t pr = 4 * i + (lane >> 3);
          asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(patch + pr * 128u + ((((uint32_t)lane & 7) ^ (pr & 7)) << 4)),
                       "r"(nxt[i].x), "r"(nxt[i].y), "r"(nxt[i].z), "r"(nxt[i].w)
                       : "memory");
        }
        if (C::kPatch) __syncwarp();
        const uint32_t cur_sf[4] = {nxt_sf.x, nxt_sf.y, nxt_sf.z, nxt_sf.w};
        // next lines: the following k-group of this item, or the first of this CTA's next item
        if (g + 1 < g1) fetch(cur_item, g + 1);
        else if (item + (int)gridDim.x < total_items) fetch(at, at.g0);
#pragma unroll
        for (int q = 0; q < 4; ++q) {                       // the four 64-wide k-steps of the group
          uint32_t cur[8];
          if constexpr (!C::kPatch) {
#pragma unroll
            for (int i = 0; i < 8; ++i) cur[i] = line[8 * q + i];
          }
#pragma unroll
          for (int c = 0; C::kPatch && c < 2; ++c)
            asm volatile("ld.shared.v4.b32 {%0, %1, %2, %3}, [%4];"
                         : "=r"(cur[4 * c]), "=r"(cur[4 * c + 1]), "=r"(cur[4 * c + 2]), "=r"(cur[4 * c + 3])
                         : "r"(patch + (uint32_t)lane * 128u + (((uint32_t)(2 * q + c) ^ sw) << 4))
                         : "memory");
          int okw = 1;
          if (lane == 0) okw = mbar_wait(bar_empty + 8 * s, ph) ? 1 : 0;
          okw = __shfl_sync(0xFFFFFFFFu, okw, 0);
          if (!okw) { if (lane == 0 && p.status) atomicCAS(p.status, 0, 125); ok = false; break; }
          const uint32_t dst = s_b + s * C::kBBytes + row_off;
          decode_half_stage(cur, cur_sf[q], dst, sw, 0);
          decode_half_stage(cur + 4, cur_sf[q] >> 16, dst, sw, 4);
          fence_async_proxy();                              // generic-proxy writes -> visible to the tensor core's reads
          __syncwarp();
          if (lane == 0) mbar_arrive(bar_full_b + 8 * s);
          if (++s == C::kStages) { s = 0; ph ^= 1; }
        }
      }
    }
  } else {
    // ------------------------------------------------------------------ epilogue: 8 warps = 2 accumulators x 4 lane quadrants
    const int quad = warp & 3;
    const int half = (warp - C::kEpiWarp0) >> 2;
    const float alpha = p.alpha ? *p.alpha : 1.0f;
    uint32_t it = 0;
    for (int item = blockIdx.x; item < total_items; item += gridDim.x, ++it) {
      const Item at = item_at(item);
      const int mt = at.tile / n_nt, nt = at.tile - mt * n_nt;
      const uint32_t buf = it % C::kAccBufs;
      int okw = 1;
      if (lane == 0) okw = mbar_wait(bar_acc_full + 8 * buf, (it / C::kAccBufs) & 1, 4 * (at.g1 - at.g0)) ? 1 : 0;
      okw = __shfl_sync(0xFFFFFFFFu, okw, 0);
      if (!okw) { if (lane == 0 && p.status) atomicCAS(p.status, 0, 124); break; }
      tc_fence_after();
      const int row = mt * 256 + half * 128 + quad * 32 + lane;
      const bool live = row < p.M;
      const uint32_t taddr = tmem + ((uint32_t)(quad * 32) << 16) + buf * 2 * BN + half * BN;
      float* partial_row = at.split < 0 ? nullptr : p.partial + (((size_t)at.split * p.tail_tiles + (at.tile - p.full_tiles)) * p.M + row) * BN;
      store_cols<BN>(p, taddr, row, live, nt * BN, alpha, partial_row, [&]() {
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(bar_acc_empty + 8 * buf);
      });
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    __syncwarp();
    tmem_dealloc<512>(tmem);
  }
}

// Tail tiles: out = bf16(alpha * sum over splits of partial[s][tile]), splits added in ascending order (reproducible).
__global__ void __launch_bounds__(256) k_w4a16_reduce(const W4A16Params p, int bn) {
  pdl_trigger();
  pdl_wait();
  const float alpha = p.alpha ? *p.alpha : 1.0f;
  const int at = ((int)blockIdx.x * (int)blockDim.x + (int)threadIdx.x) * 4;             // four columns of a tile's row
  const int t = (int)blockIdx.y;
  const int row = at / bn, col = (p.full_tiles + t) * bn + at % bn;
  if (row < p.M) {
    const float* src = p.partial + (size_t)t * p.M * bn + at;
    float4 acc = *reinterpret_cast<const float4*>(src);
    for (int s = 1; s < p.splits; ++s) {
      const float4 v = *reinterpret_cast<const float4*>(src + (size_t)s * p.tail_tiles * p.M * bn);
      acc.x += v.x; acc.y += v.y; acc.z += v.z; acc.w += v.w;
    }
    const __nv_bfloat162 lo = __floats2bfloat162_rn(acc.x * alpha, acc.y * alpha), hi = __floats2bfloat162_rn(acc.z * alpha, acc.w * alpha);
    uint2 o;
    o.x = *reinterpret_cast<const uint32_t*>(&lo);
    o.y = *reinterpret_cast<const uint32_t*>(&hi);
    *reinterpret_cast<uint2*>(p.out + (size_t)row * p.out_stride + col) = o;
  }
}

}  // namespace

// Tile width and, up to 128 rows, the split of the last wave. The tiles left over after whole waves are shared by as many CTAs as
// the SMs hold (at most eight, at least one k-group each). Behind whole waves that pays for its partial tiles and the second launch
// only when a tile is long: from 16 k-groups on. The plan of a batch of 17 to 128 rows does not depend on its rows, so a row has
// one value in all of them. Above, which tiles end up in the last wave depends on the batch: a split there would give a row other
// last bits at another position, so there is none, which gives up time (8192 x 4096 x 12288 696 us with a split, 759 without;
// 129 x 4096 x 4096 23 and 42). `room`: the caller has a workspace for the partial tiles.
struct W4A16Plan {
  int bn, full_tiles, tail_tiles, splits;
};
static W4A16Plan w4a16_plan(int64_t m, int64_t n, int64_t k, int sms, bool room) {
  W4A16Plan pl;
  // Up to 128 rows half of a wide tile's accumulators idle: it pays when the tiles are long and fill the device, by their number
  // (M = 64, N = 25600, K = 8192: 120 us against 158) or by a split that there is room for (M = 64, N = 4096, K = 12288: 31 us against
  // 36; N = 2048, K = 4096: 16 against 12). A split that falls away leaves half as many CTAs as narrow tiles do (M = 64, N = 4096,
  // K = 8192: 116 us against 81; M = 128, N = 8192, K = 12288: 179 against 120). Above 128 rows narrow tiles are the better ones while
  // all of them run at once: half the work of a wide tile each, and no trip through the patch that a single tile per SM cannot hide
  // (129 x 4096 x 4096 63 us wide, 42 narrow; 1000 x 4096 x 4096, the last of that width, 61 and 45; 1200 rows 63 wide). Both widths
  // add in the same order.
  pl.bn = (m > 128 ? w4a16_wide_tiles(m, n, sms) : n % 256 == 0 && room && n >= 4096 && k >= 8192) ? 256 : 128;
  const int64_t tiles = (m + 255) / 256 * (n / pl.bn), groups = k / 256, tail = tiles % sms;
  int64_t s = tail ? sms / tail : 1;
  if (s > 8) s = 8;
  if (s > groups) s = groups;
  if (s < 2 || !room || m > 128 || w4a16_decode_wins(m, n, k) || (tiles > tail && groups < 16)) s = 1;
  pl.splits = (int)s;
  pl.tail_tiles = s > 1 ? (int)tail : 0;
  pl.full_tiles = (int)(tiles - pl.tail_tiles);
  return pl;
}
static int64_t w4a16_partial_bytes(const W4A16Plan& pl, int64_t m) { return (int64_t)pl.splits * pl.tail_tiles * m * pl.bn * 4; }

int64_t gemm_w4a16_workspace_bytes(int64_t m, int64_t n, int64_t k) {
  return w4a16_expand_wins(m, n, k) ? n * k * 2 : w4a16_partial_bytes(w4a16_plan(m, n, k, sm_count(), true), m);
}

template <int BN>
static int launch_w4a16(const CUtensorMap& ta, const W4A16Params& p, int sms, cudaStream_t st) {
  auto kern = k_gemm_w4a16<BN>;
  static SmemOptIn opt_in;
  if (int e = opt_in.ensure(kern, WCfg<BN>::kSmem)) return e;
  const int64_t items = (int64_t)p.full_tiles + (int64_t)p.tail_tiles * p.splits;
  return (int)launch_chain(kern, dim3((unsigned)(items < sms ? items : sms)), dim3(WCfg<BN>::kThreads), WCfg<BN>::kSmem, st, ta, p);
}

int launch_gemm_w4a16(const void* a, int64_t a_stride, const void* b_q, const void* b_sf, const float* alpha, int64_t m, int64_t n,
                      int64_t k, void* out, int64_t out_stride, void* workspace, int64_t workspace_bytes, int32_t* status,
                      cudaStream_t st) {
  if (m == 0) return 0;
  if (w4a16_expand_room(workspace, workspace_bytes, n, k) && w4a16_expand_wins(m, n, k))
    return launch_gemm_w4a16_expand(a, a_stride, b_q, b_sf, alpha, m, n, k, out, out_stride, workspace, status, st);
  const int sms = sm_count();
  W4A16Plan pl = w4a16_plan(m, n, k, sms, true);
  const bool no_room = pl.splits > 1 && (!workspace || workspace_bytes < w4a16_partial_bytes(pl, m));
  // workspace_bytes < 0: one sum in ascending k per element at every size, so the tile kernel, unsplit
  if (workspace_bytes >= 0 && m <= kW4A16DecodeMaxM && (no_room || w4a16_decode_wins(m, n, k)))
    return launch_gemm_w4a16_decode(a, a_stride, b_q, b_sf, alpha, m, n, k, out, out_stride, st);
  if (no_room) pl = w4a16_plan(m, n, k, sms, false);
  const int bn = pl.bn;
  CUtensorMap ta;
  int rc = make_operand_map(&ta, a, (uint64_t)m, (uint64_t)k * 2, 256, (uint64_t)a_stride * 2);
  if (rc) return rc;
  W4A16Params p;
  p.b_q = (const uint8_t*)b_q;
  p.b_sf = (const uint8_t*)b_sf;
  p.alpha = alpha;
  p.out = (__nv_bfloat16*)out;
  p.out_stride = out_stride;
  p.M = (int)m;
  p.N = (int)n;
  p.K = (int)k;
  p.status = status;
  p.partial = (float*)workspace;
  p.groups_per_split = (int)((k / 256 + pl.splits - 1) / pl.splits);
  p.splits = (int)((k / 256 + p.groups_per_split - 1) / p.groups_per_split);              // no empty split
  p.full_tiles = pl.full_tiles;
  p.tail_tiles = pl.tail_tiles;
  rc = bn == 256 ? launch_w4a16<256>(ta, p, sms, st) : launch_w4a16<128>(ta, p, sms, st);
  if (rc || p.splits == 1) return rc;
  const int64_t quads = m * (bn / 4);
  return (int)launch_chain(k_w4a16_reduce, dim3((unsigned)((quads + 255) / 256), (unsigned)p.tail_tiles), dim3(256), 0, st, p, bn);
}

}  // namespace b200
