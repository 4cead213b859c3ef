// Dense GEMM with bf16 activations and NVFP4 weights for many tokens (prefill): out = bf16(alpha * A @ decode(B)^T), the same
// contract as gemm_w4a16.cu (gemm/dense/bf16_nvfp4_gemm/problem/reference.py:10-15), in two launches.
//
// The tile kernel of gemm_w4a16.cu decodes a weight row again for every 256 rows of A, and its decoders share an SM's issue slots
// and shared-memory ports with the operand traffic. Unless there are few rows for very many weights, or K is short, it is cheaper from 129
// rows on (w4a16_expand_wins) to expand the weights ONCE into a bf16 scratch (k_w4a16_expand, exact: bound by its 2 written bytes a
// weight) and to run the product as a pure bf16 GEMM (k_gemm_bf16_pair, tensor-bound) that has nothing but TMA, MMAs and an
// overlapped epilogue in it.
//
// k_gemm_bf16_pair: a cluster of two CTAs drives tcgen05.mma.cta_group::2 on 256 x 256 tiles, so each SM fetches 128 rows of A and
// 128 of B per 64-wide k-step (32 KB for 512 tensor cycles). Seven stages; two 256-column accumulators fill TMEM, so a tile's
// epilogue runs beside the next tile's k-loop.
// Both launches are in plain stream order, not programmatic. A programmatic form of the two, ten calls of 129 x 4096 x 12288 back to back,
// did not finish, and no bounded wait expired in it. The cause was not found. By the rule that a dependent grid starts only when every
// block before it has triggered or ended, no block can have been kept out. If that rule failed for clusters, then only through blocks
// of the NEXT expansion, let in by the GEMM's trigger and waiting on the SMs (several waves of them) while clusters still looked
// for room: that GEMM has 64 blocks, so waiting clusters of its own left 84 SMs to the expansion before it.
// Here nothing is let in early, and no cluster kernel of the library triggers (launch_clusters in kernels.cuh).
// Additions per element run in ascending k like the tile kernel's: same bits.
#include "kernels.cuh"
#include "ptx.cuh"
#include "w4a16.cuh"

namespace b200 {

namespace {

// ----------------------------------------------------------------------------- expansion
// One thread expands kExpandUnits blocks of 16 weights: 8 payload bytes and one scale byte in, one 32-byte sector out each. The
// loads of all units are issued before the first store.
constexpr int kExpandThreads = 256;
constexpr int kExpandUnits = 4;

__global__ void __launch_bounds__(kExpandThreads) k_w4a16_expand(const uint2* __restrict__ q, const uint8_t* __restrict__ sf, int64_t blocks,
                                                                 uint8_t* __restrict__ out) {
  const int64_t first = (int64_t)blockIdx.x * (kExpandThreads * kExpandUnits) + threadIdx.x;
  uint2 w[kExpandUnits];
  uint32_t s[kExpandUnits];
#pragma unroll
  for (int i = 0; i < kExpandUnits; ++i) {
    const int64_t b = first + i * kExpandThreads;
    w[i] = b < blocks ? __ldg(q + b) : make_uint2(0u, 0u);
    s[i] = b < blocks ? __ldg(sf + b) : 0u;
  }
#pragma unroll
  for (int i = 0; i < kExpandUnits; ++i) {
    const int64_t b = first + i * kExpandThreads;
    const uint32_t sc = __byte_perm(e4m3x2_to_bf16x2(s[i]), 0, 0x1010);
    uint32_t o[8];
    e2m1x4_to_bf16x2(w[i].x, o[0], o[1]);
    e2m1x4_to_bf16x2(w[i].x >> 16, o[2], o[3]);
    e2m1x4_to_bf16x2(w[i].y, o[4], o[5]);
    e2m1x4_to_bf16x2(w[i].y >> 16, o[6], o[7]);
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      const __nv_bfloat162 prod = __hmul2(*reinterpret_cast<const __nv_bfloat162*>(&o[j]), *reinterpret_cast<const __nv_bfloat162*>(&sc));
      o[j] = *reinterpret_cast<const uint32_t*>(&prod);
    }
    if (b < blocks)
      asm volatile("st.global.v8.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};" ::"l"(out + b * 32), "r"(o[0]), "r"(o[1]), "r"(o[2]), "r"(o[3]),
                   "r"(o[4]), "r"(o[5]), "r"(o[6]), "r"(o[7])
                   : "memory");
  }
}

// ----------------------------------------------------------------------------- bf16 GEMM on CTA pairs
template <int BN>
struct BpCfg {
  static constexpr int kStages = BN == 256 ? 7 : 9;
  static constexpr int kABytes = 128 * 128;                 // per CTA: 128 rows x 64 bf16
  static constexpr int kBBytes = BN / 2 * 128;              // per CTA: half of the tile's weight rows
  static constexpr int kStageBytes = kABytes + kBBytes;
  static constexpr int kSmem = kStages * kStageBytes + 1024 + 256;
  static_assert(kSmem <= 232448 && 16 * kStages + 36 <= 256, "shared memory");
};
constexpr int kBpEpiWarps = 8;                              // two column halves x four lane quadrants
constexpr int kBpThreads = 32 * (2 + kBpEpiWarps);
constexpr int kBpGroup = 8;                                 // m-tiles of a raster group

struct BpParams {
  const float* alpha;       // device scalar or null (= 1)
  __nv_bfloat16* out;
  int64_t out_stride;
  int M, N, K;
  int32_t* status;
};

DEV void mma_bf16_pair(uint32_t d_tmem, uint64_t a_desc, uint64_t b_desc, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n\t}"
      ::"r"(d_tmem), "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(accumulate)
      : "memory");
}

// Tiles in groups of kBpGroup m-tiles, m fastest inside a group: the pairs of a wave cover a compact block of the output, so its
// operand rows are read from HBM a few times in all.
DEV void bp_tile(int t, int n_mt, int n_nt, int& mt, int& nt) {
  const int per = kBpGroup * n_nt, g = t / per, r = t - g * per;
  const int rows = min(kBpGroup, n_mt - g * kBpGroup);
  nt = r / rows;
  mt = g * kBpGroup + (r - nt * rows);
}

template <int BN>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(kBpThreads, 1)
k_gemm_bf16_pair(const __grid_constant__ CUtensorMap tm_a, const __grid_constant__ CUtensorMap tm_b, const BpParams p) {
  using C = BpCfg<BN>;
  extern __shared__ uint8_t smem_raw[];
  const uint32_t base = (smem_u32(smem_raw) + 1023u) & ~1023u;
  const uint32_t s_a = base, s_b = s_a + C::kStages * C::kABytes;
  const uint32_t bar_full = s_b + C::kStages * C::kBBytes;     // leader: two producer arrivals and both CTAs' bytes
  const uint32_t bar_empty = bar_full + 8 * C::kStages;        // both CTAs: MMAs of the stage retired
  const uint32_t bar_acc_full = bar_empty + 8 * C::kStages;    // [2] both CTAs
  const uint32_t bar_acc_empty = bar_acc_full + 16;           // [2] leader: the pair's epilogue warps
  const uint32_t s_slot = bar_acc_empty + 16;
  const int warp = warp_uniform();
  const int lane = threadIdx.x & 31;
  const uint32_t rank = cluster_ctarank();

  if (threadIdx.x == 0) {
    for (int s = 0; s < C::kStages; ++s) {
      mbar_init(bar_full + 8 * s, 2);
      mbar_init(bar_empty + 8 * s, 1);
    }
    for (int b = 0; b < 2; ++b) {
      mbar_init(bar_acc_full + 8 * b, 1);
      mbar_init(bar_acc_empty + 8 * b, 2 * kBpEpiWarps);
    }
    mbar_init_fence();
    tma_prefetch_desc(&tm_a);
    tma_prefetch_desc(&tm_b);
  }
  if (warp == 1) tmem_alloc_pair<512>(s_slot);
  tc_fence_before();
  __syncthreads();
  cluster_sync_all();
  tc_fence_after();
  uint32_t tmem;
  asm volatile("ld.shared.u32 %0, [%1];" : "=r"(tmem) : "r"(s_slot));

  const int n_mt = (p.M + 255) / 256, n_nt = (p.N + BN - 1) / BN, nk = p.K / 64;
  const int tiles = n_mt * n_nt;
  const int first = blockIdx.x >> 1, stride = gridDim.x >> 1;

  if (warp == 0) {
    // ------------------------------------------------------------------ TMA producer (each CTA its own halves)
    if (elect_one()) {
      uint32_t s = 0, ph = 1;
      bool ok = true;
      const uint32_t full0 = map_to_cta(bar_full, 0);
      for (int t = first; ok && t < tiles; t += stride) {
        int mt, nt;
        bp_tile(t, n_mt, n_nt, mt, nt);
        const int row_a = mt * 256 + (int)rank * 128, row_b = nt * BN + (int)rank * (BN / 2);   // rows past the end read as zeros
        for (int ks = 0; ks < nk; ++ks) {
          if (!mbar_wait_cluster(bar_empty + 8 * s, ph)) { if (p.status) atomicCAS(p.status, 0, 131); ok = false; break; }
          const uint32_t full = full0 + 8 * s;
          mbar_expect_tx_remote(full, C::kStageBytes);
          tma_load_2d_pair(s_a + s * C::kABytes, &tm_a, full, ks * 128, row_a);
          tma_load_2d_pair(s_b + s * C::kBBytes, &tm_b, full, ks * 128, row_b);
          if (++s == C::kStages) { s = 0; ph ^= 1; }
        }
      }
    }
    __syncwarp();
  } else if (warp == 1) {
    // ------------------------------------------------------------------ MMA issuer (leader)
    if (rank == 0 && elect_one()) {
      constexpr uint32_t idesc = make_idesc_bf16(256, BN);
      constexpr uint32_t kHiOp = (1024u >> 4) | (1u << 14) | (2u << 29);   // SBO 1024, version 1, SWIZZLE_128B
      const uint32_t a_lo0 = ((s_a >> 4) & 0x3FFF) | (1u << 16), b_lo0 = ((s_b >> 4) & 0x3FFF) | (1u << 16);
      uint32_t s = 0, ph = 0, it = 0;
      bool ok = true;
      for (int t = first; ok && t < tiles; t += stride, ++it) {
        const uint32_t buf = it & 1;
        if (!mbar_wait_cluster(bar_acc_empty + 8 * buf, ((it >> 1) & 1) ^ 1)) { if (p.status) atomicCAS(p.status, 0, 132); break; }
        tc_fence_after();
        const uint32_t acc = tmem + buf * BN;
        for (int ks = 0; ks < nk; ++ks) {
          if (!mbar_wait_cluster(bar_full + 8 * s, ph)) { if (p.status) atomicCAS(p.status, 0, 133); ok = false; break; }
          tc_fence_after();
          const uint32_t a_lo = a_lo0 + s * (C::kABytes >> 4), b_lo = b_lo0 + s * (C::kBBytes >> 4);
#pragma unroll
          for (int q = 0; q < 4; ++q)
            mma_bf16_pair(acc, ((uint64_t)kHiOp << 32) | (a_lo + 2 * q), ((uint64_t)kHiOp << 32) | (b_lo + 2 * q), idesc, (ks | q) ? 1u : 0u);
          mma_commit_pair(bar_empty + 8 * s);
          if (++s == C::kStages) { s = 0; ph ^= 1; }
        }
        if (ok) mma_commit_pair(bar_acc_full + 8 * buf);
      }
    }
    __syncwarp();
  } else {
    // ------------------------------------------------------------------ epilogue: own 128 rows x BN columns
    const int quad = warp & 3, half = (warp - 2) >> 2;
    const float alpha = p.alpha ? *p.alpha : 1.0f;
    const uint32_t acc_empty0 = map_to_cta(bar_acc_empty, 0);
    uint32_t it = 0;
    for (int t = first; t < tiles; t += stride, ++it) {
      int mt, nt;
      bp_tile(t, n_mt, n_nt, mt, nt);
      const uint32_t buf = it & 1;
      int okw = 1;
      if (lane == 0) okw = mbar_wait_cluster(bar_acc_full + 8 * buf, (it >> 1) & 1, nk) ? 1 : 0;
      okw = __shfl_sync(0xFFFFFFFFu, okw, 0);
      if (!okw) { if (lane == 0 && p.status) atomicCAS(p.status, 0, 134); break; }
      tc_fence_after();
      const int row = mt * 256 + (int)rank * 128 + quad * 32 + lane, col0 = nt * BN + half * (BN / 2);
      const bool live = row < p.M && col0 < p.N;              // N is a multiple of 128
      if (__any_sync(0xFFFFFFFFu, live)) {
        const uint32_t taddr = tmem + ((uint32_t)(quad * 32) << 16) + buf * BN + half * (BN / 2);
        __nv_bfloat16* dst = p.out + (size_t)row * p.out_stride + col0;
#pragma unroll
        for (int col = 0; col < BN / 2; col += 64) {
          float v[2][32];
          tmem_ld32(taddr + col, v[0]);
          tmem_ld32(taddr + col + 32, v[1]);
          tmem_ld_wait();
          if (live) {
#pragma unroll
            for (int cb = 0; cb < 2; ++cb) {
              uint32_t o[16];
#pragma unroll
              for (int j = 0; j < 16; ++j) {
                const __nv_bfloat162 pr = __floats2bfloat162_rn(v[cb][2 * j] * alpha, v[cb][2 * j + 1] * alpha);
                o[j] = *reinterpret_cast<const uint32_t*>(&pr);
              }
              __nv_bfloat16* d = dst + col + cb * 32;
#pragma unroll
              for (int j = 0; j < 2; ++j)
                asm volatile("st.global.L1::no_allocate.v8.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};" ::"l"(d + 16 * j), "r"(o[8 * j]),
                             "r"(o[8 * j + 1]), "r"(o[8 * j + 2]), "r"(o[8 * j + 3]), "r"(o[8 * j + 4]), "r"(o[8 * j + 5]),
                             "r"(o[8 * j + 6]), "r"(o[8 * j + 7])
                             : "memory");
            }
          }
        }
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive_remote(acc_empty0 + 8 * buf);
    }
  }
  tc_fence_before();
  __syncthreads();
  cluster_sync_all();
  if (warp == 1) {
    __syncwarp();
    tmem_dealloc_pair<512>(tmem);
  }
}

template <int BN>
int launch_bp(const CUtensorMap& ta, const CUtensorMap& tb, const BpParams& p, int pairs, cudaStream_t st) {
  auto kern = k_gemm_bf16_pair<BN>;
  static SmemOptIn opt_in;
  if (int e = opt_in.ensure(kern, BpCfg<BN>::kSmem)) return e;
  const int64_t tiles = ((int64_t)p.M + 255) / 256 * ((p.N + BN - 1) / BN);
  kern<<<dim3((unsigned)(2 * (tiles < pairs ? tiles : pairs))), dim3(kBpThreads), BpCfg<BN>::kSmem, st>>>(ta, tb, p);
  return (int)cudaGetLastError();
}

// 128-wide tiles while their waves of pairs are fewer than 1 / 0.57 of the wide ones': half the work at a little more than half of the
// time each (their stage moves 24 KB for 256 tensor cycles). Wide / narrow: 256 x 4096 x 12288, one wave each, 97 / 67 us with the
// expansion; 1536 rows, 2 and 3 waves, 150 / 135; 2048 rows, 2 and 4 waves, 158 / 172; 8192 rows, 7 and 14 waves, 543 / 612. 64-wide
// tiles were no faster anywhere than 128-wide ones (129 x 1280 x 12288 42 us both).
int bp_tile_n(int64_t m, int64_t n, int pairs) {
  const auto waves = [&](int bn) { return ((m + 255) / 256 * ((n + bn - 1) / bn) + pairs - 1) / pairs; };
  return waves(128) * 57 < waves(256) * 100 ? 128 : 256;
}

}  // namespace

// Where the two launches are the faster way: by the time that each way takes, in microseconds of a call among others. Both are waves of
// tiles, a wave a few microseconds and the k-steps of 64 of one tile, a step the slower the fuller the wave; the expansion adds its
// launches and the bytes of the weights, more for each beyond what stays in L2. Fitted to 2544 shapes (128 <= N <= 65536,
// 256 <= K <= 28672, 129 <= M <= 8192, both ways timed): choosing by it costs 0.05 % against always taking the faster way, and where it
// takes the expansion that is at most 9 % slower than the tile kernel. (Tile kernel / here: 256 x 4096 x 4096 43 / 25 us, 1024 x 2048 x 8192
// 82 / 36, 8192 x 4096 x 12288 774 / 560; few rows for very many weights 129 x 16384 x 4096 44 / 62, 200 x 28672 x 2048 39 / 72; a
// short K 2048 x 2048 x 1024 14.7 / 16.7.) With one k-group of 256 there is nothing to save. In a graph, where the two launches cost 4 us
// less, the expansion would win from shorter loops on (2048 x 2048 x 1024 14.6 / 12.6); the rule is for separate calls. Both ways give
// the same bits.
bool w4a16_expand_wins(int64_t m, int64_t n, int64_t k) {
  if (m <= 128 || k < 512 || n * k * 2 > kW4A16ExpandMax) return false;
  const int sms = sm_count(), pairs = sms / 2;
  const double steps = (double)(k / 64), mega = (double)(n * k) * 1e-6;
  const bool wide = w4a16_wide_tiles(m, n, sms);
  const int64_t tiles = (m + 255) / 256 * (n / (wide ? 256 : 128)), waves = (tiles + sms - 1) / sms;
  const double tile_us = 2.0 + waves * (2.2 + steps * (wide ? 1.08 : 0.595 + 0.084 * tiles / (waves * sms)));
  const int bn = bp_tile_n(m, n, pairs);
  const int64_t pair_tiles = (m + 255) / 256 * ((n + bn - 1) / bn), pair_waves = (pair_tiles + pairs - 1) / pairs;
  const double expand_us = 10.2 + 0.294 * mega + (mega > 20 ? 0.267 * (mega - 20) : 0);
  return expand_us + pair_waves * (1.45 + steps * (bn == 256 ? 0.186 + 0.15 * pair_tiles / (pair_waves * pairs) : 0.141)) < tile_us;
}

int launch_gemm_w4a16_expand(const void* a, int64_t a_stride, const void* b_q, const void* b_sf, const float* alpha, int64_t m, int64_t n,
                             int64_t k, void* out, int64_t out_stride, void* scratch, int32_t* status, cudaStream_t st) {
  const int64_t blocks = n * (k / 16), per = kExpandThreads * kExpandUnits;
  k_w4a16_expand<<<dim3((unsigned)((blocks + per - 1) / per)), dim3(kExpandThreads), 0, st>>>((const uint2*)b_q, (const uint8_t*)b_sf,
                                                                                              blocks, (uint8_t*)scratch);
  int rc = (int)cudaGetLastError();
  if (rc) return rc;
  const int pairs = sm_count() / 2;
  const int bn = bp_tile_n(m, n, pairs);
  CUtensorMap ta, tb;
  rc = make_operand_map(&ta, a, (uint64_t)m, (uint64_t)k * 2, 128, (uint64_t)a_stride * 2);
  if (!rc) rc = make_operand_map(&tb, scratch, (uint64_t)n, (uint64_t)k * 2, (uint32_t)bn / 2);
  if (rc) return rc;
  BpParams p;
  p.alpha = alpha;
  p.out = (__nv_bfloat16*)out;
  p.out_stride = out_stride;
  p.M = (int)m;
  p.N = (int)n;
  p.K = (int)k;
  p.status = status;
  return bn == 256 ? launch_bp<256>(ta, tb, p, pairs, st) : launch_bp<128>(ta, tb, p, pairs, st);
}

}  // namespace b200
