// Dense GEMM with bf16 activations and NVFP4 weights for a handful of tokens (decode): out = bf16(alpha * A @ decode(B)^T),
// the same contract as gemm_w4a16.cu (gemm/dense/bf16_nvfp4_gemm/problem/reference.py:10-15).
//
// With few tokens the product is a stream over the weights (N * K * 9/16 bytes). The tile kernel serves it badly: its decoder
// threads hold one 128-byte line each and hand every decoded weight through shared memory to a 256-row MMA that is almost
// all padding. Here the weights never leave the registers: a warp decodes 64 weight rows straight into the A fragments of
// mma.sync.m16n8k16 (weight rows = M side, tokens = N side, so 8 tokens are no padding). What bounds it is the decode's issue
// rate, the weight stream and, from 16 tokens on, the activation fragments' trips through shared memory, a few us each at
// N = 4096, K = 12288.
//
// K order: a dot product may take its k in any order as long as both operands agree. Lane (g, t) of a warp (g = lane / 4,
// t = lane % 4) therefore reads 32 CONSECUTIVE weights of rows g, g + 8, .. g + 56 per 128-wide unit of K (16 payload bytes
// and two scale bytes each) and the same 32 activations of token g, and an MMA step multiplies whatever four k's the lane has
// there. Activations pass through a warp-private shared-memory tile: read from global memory a token row at a time (256
// contiguous bytes; fetched by the fragments' own addresses a load touches 32 lines), kept in fragment order.
//
// Split: 8 warps of a block take the units of K in turn, and a cluster of C blocks splits K further while (N / 64) * C blocks
// are resident at once: two per SM up to 16 tokens, one above (255 registers). Partial sums meet in shared memory, then in distributed shared memory, each time in a fixed order
// (reproducible, no workspace, one launch).
#include "kernels.cuh"
#include "ptx.cuh"

namespace b200 {

namespace {

constexpr int kDecWarps = 8;
constexpr int kDecRows = 64;                 // weight rows of a block (every warp computes all of them over its share of K)
constexpr int kDecUnit = 128;                // K of one step of a warp
constexpr int kDecPitch = kDecRows + 4;      // floats between tokens of a partial tile: conflict-free fragment stores

// Two E4M3 bytes (low 16 bits of s) -> bf16x2 of scale * 2^118.
DEV uint32_t scale_pair(uint32_t s) {
  uint32_t h;
  asm("{\n\t.reg .b16 t;\n\tcvt.u16.u32 t, %1;\n\tcvt.rn.f16x2.e4m3x2 %0, t;\n\t}" : "=r"(h) : "r"(s & 0xFFFFu));
  const float2 f = __half22float2(*reinterpret_cast<const __half2*>(&h));
  const __nv_bfloat162 b = __floats2bfloat162_rn(f.x * 0x1p118f, f.y * 0x1p118f);
  return *reinterpret_cast<const uint32_t*>(&b);
}

// Elements k and k + 4 of a payload word (nibble k of both 16-bit halves) -> bf16x2 of weight * 2^-126. The nibble's e, e, m
// bits placed at bits 8..6 of a bf16 ARE the weight times 2^-126, the subnormal 0.5 included; the block scale carries 2^118
// (448 * 2^118 still fits bf16), so the product is weight * scale * 2^-8, exact in bf16, and the epilogue takes the 2^-8 back.
template <int Kk>
DEV uint32_t weight_pair(uint32_t w, uint32_t scale2) {
  constexpr int kUp = 12 - 4 * Kk;                             // sign bit 4k + 3 -> 15
  const uint32_t sg = (w << kUp) & 0x80008000u;
  const uint32_t mag = (Kk >= 2 ? w >> (4 * Kk - 6) : w << (6 - 4 * Kk)) & 0x01C001C0u;
  const uint32_t v = sg | mag;
  const __nv_bfloat162 p = __hmul2(*reinterpret_cast<const __nv_bfloat162*>(&v), *reinterpret_cast<const __nv_bfloat162*>(&scale2));
  return *reinterpret_cast<const uint32_t*>(&p);
}

DEV void mma_m16n8k16(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
  asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
               : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
               : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

// NT = groups of eight tokens (M <= 8 * NT).
template <int NT>
constexpr int dec_smem_bytes() {
  const int x = kDecWarps * NT * 8 * kDecUnit * 2, part = kDecWarps * 8 * NT * kDecPitch * 4;
  return x > part ? x : part;
}

// Blocks an SM holds: the fragments of 32 tokens take 255 registers a thread.
template <int NT>
constexpr int dec_blocks_per_sm() { return NT <= 2 ? 2 : 1; }

template <int NT>
__global__ void __launch_bounds__(32 * kDecWarps, dec_blocks_per_sm<NT>())
k_gemm_w4a16_decode(const __nv_bfloat16* __restrict__ a, int64_t a_stride, const uint8_t* __restrict__ b_q,
                    const uint8_t* __restrict__ b_sf, const float* __restrict__ alpha_ptr, __nv_bfloat16* __restrict__ out,
                    int64_t out_stride, int M, int K, int split) {
  extern __shared__ uint4 dec_smem[];                          // activation tiles of the warps, later their partial sums
  constexpr int kPart = 8 * NT * kDecPitch;                    // floats of one warp's partial tile
  float* part = reinterpret_cast<float*>(dec_smem);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int g = lane >> 2, t = lane & 3;
  const int rank = (int)blockIdx.x % split;                    // == rank in the cluster
  const int64_t row0 = (int64_t)((int)blockIdx.x / split) * kDecRows;
  const int units = K / kDecUnit;
  uint4* xs = dec_smem + warp * (NT * 8 * kDecUnit * 2 / 16);  // [NT][4 words of a lane][8 tokens x 4 lanes] 16-byte pieces
  if (split == 1) pdl_trigger();                               // never from a cluster (launch_clusters)
  pdl_wait();

  float acc[4][NT][4];
#pragma unroll
  for (int mt = 0; mt < 4; ++mt)
#pragma unroll
    for (int n = 0; n < NT; ++n)
#pragma unroll
      for (int i = 0; i < 4; ++i) acc[mt][n][i] = 0.f;

  for (int u = rank * kDecWarps + warp; u < units; u += split * kDecWarps) {
    uint4 w[8];                                                // rows g + 8r
    uint32_t sf[8];
#pragma unroll
    for (int r = 0; r < 8; ++r) {
      const int64_t row = row0 + g + 8 * r;
      w[r] = __ldg(reinterpret_cast<const uint4*>(b_q + row * (K >> 1) + u * 64 + t * 16));
      sf[r] = __ldg(reinterpret_cast<const unsigned short*>(b_sf + row * (K >> 4) + u * 8 + t * 2));
    }
    // piece (token, kc): 8 activations of lane kc / 4's word kc % 4; the XOR spreads a store's lanes over the banks
    __syncwarp();
#pragma unroll
    for (int i0 = 0; i0 < 4 * NT; i0 += 8) {
      uint4 x[8];
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        const int tok = (i0 + i) * 2 + (lane >> 4);
        x[i] = make_uint4(0u, 0u, 0u, 0u);
        if (i0 + i < 4 * NT && tok < M) x[i] = __ldg(reinterpret_cast<const uint4*>(a + (int64_t)tok * a_stride + u * kDecUnit) + (lane & 15));
      }
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        const int tok = (i0 + i) * 2 + (lane >> 4), word = lane & 3, tq = (lane & 15) >> 2;
        if (i0 + i < 4 * NT) xs[((tok >> 3) * 4 + word) * 32 + (((tok & 7) * 4 + tq) ^ (word << 1))] = x[i];
      }
    }
    __syncwarp();
    uint32_t sc[8];
#pragma unroll
    for (int r = 0; r < 8; ++r) sc[r] = scale_pair(sf[r]);
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      uint32_t xb[NT][4];
#pragma unroll
      for (int n = 0; n < NT; ++n) {                           // pairs (x_k, x_{k+4}) to match the weight pairs
        const uint4 x = xs[(n * 4 + j) * 32 + (lane ^ (j << 1))];
        xb[n][0] = __byte_perm(x.x, x.z, 0x5410);
        xb[n][1] = __byte_perm(x.x, x.z, 0x7632);
        xb[n][2] = __byte_perm(x.y, x.w, 0x5410);
        xb[n][3] = __byte_perm(x.y, x.w, 0x7632);
      }
#pragma unroll
      for (int mt = 0; mt < 4; ++mt) {
        const uint4 wa = w[2 * mt], wb = w[2 * mt + 1];
        const uint32_t w0 = j == 0 ? wa.x : j == 1 ? wa.y : j == 2 ? wa.z : wa.w, w1 = j == 0 ? wb.x : j == 1 ? wb.y : j == 2 ? wb.z : wb.w;
        const uint32_t c0 = __byte_perm(sc[2 * mt], 0, (j & 2) ? 0x3232 : 0x1010), c1 = __byte_perm(sc[2 * mt + 1], 0, (j & 2) ? 0x3232 : 0x1010);
        const uint32_t a00 = weight_pair<0>(w0, c0), a01 = weight_pair<0>(w1, c1), a02 = weight_pair<1>(w0, c0), a03 = weight_pair<1>(w1, c1);
        const uint32_t a10 = weight_pair<2>(w0, c0), a11 = weight_pair<2>(w1, c1), a12 = weight_pair<3>(w0, c0), a13 = weight_pair<3>(w1, c1);
#pragma unroll
        for (int n = 0; n < NT; ++n) {
          mma_m16n8k16(acc[mt][n], a00, a01, a02, a03, xb[n][0], xb[n][1]);
          mma_m16n8k16(acc[mt][n], a10, a11, a12, a13, xb[n][2], xb[n][3]);
        }
      }
    }
  }
  __syncthreads();                                             // the activation tiles are done with
  // accumulator (row g / g + 8 of m-tile mt, tokens 8n + 2t, 8n + 2t + 1) -> partial tile [token][row]
#pragma unroll
  for (int mt = 0; mt < 4; ++mt)
#pragma unroll
    for (int n = 0; n < NT; ++n)
#pragma unroll
      for (int i = 0; i < 4; ++i)
        part[warp * kPart + (8 * n + 2 * t + (i & 1)) * kDecPitch + 16 * mt + g + 8 * (i >> 1)] = acc[mt][n][i];
  __syncthreads();
  const float scale = 256.0f;
  const float alpha = alpha_ptr ? *alpha_ptr : 1.0f;
  const int outputs = M * kDecRows;
  if (split == 1) {
    for (int i = threadIdx.x; i < outputs; i += 32 * kDecWarps) {
      const int tok = i / kDecRows, row = i % kDecRows;
      float sum = part[tok * kDecPitch + row];
#pragma unroll
      for (int w = 1; w < kDecWarps; ++w) sum += part[w * kPart + tok * kDecPitch + row];
      out[tok * out_stride + row0 + row] = __float2bfloat16_rn((sum * scale) * alpha);
    }
    return;
  }
  for (int i = threadIdx.x; i < outputs; i += 32 * kDecWarps) {
    const int at = (i / kDecRows) * kDecPitch + i % kDecRows;
    float sum = part[at];
#pragma unroll
    for (int w = 1; w < kDecWarps; ++w) sum += part[w * kPart + at];
    part[at] = sum;                                            // each position belongs to one thread
  }
  cluster_sync_all();                                          // every block's sums are in place
  const uint32_t base = smem_u32(part);
  for (int i = rank * 32 * kDecWarps + threadIdx.x; i < outputs; i += split * 32 * kDecWarps) {
    const int tok = i / kDecRows, row = i % kDecRows;
    const uint32_t at = base + (uint32_t)(tok * kDecPitch + row) * 4u;
    float v[8];
#pragma unroll
    for (int r = 0; r < 8; ++r) {
      v[r] = 0.f;
      if (r < split) asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v[r]) : "r"(map_to_cta(at, (uint32_t)r)));
    }
    float sum = v[0];
#pragma unroll
    for (int r = 1; r < 8; ++r)
      if (r < split) sum += v[r];
    out[tok * out_stride + row0 + row] = __float2bfloat16_rn((sum * scale) * alpha);
  }
  cluster_sync_all();                                          // nobody leaves while a peer still reads its sums
}

// Blocks per row tile: double while all are resident at once and the added blocks would have K to work on. Counting two per SM
// for 32 tokens, of which one is resident, made two uneven waves of clusters (32 x 2048 x 7168 22.4 us against 12.4 with one). With
// one block per SM the GPCs do not hold as many clusters of eight as there are SMs for, so those stop at half the device.
int dec_split(int64_t n, int64_t k, int per_sm) {
  const int64_t tiles = n / kDecRows, units = k / kDecUnit, slots = (int64_t)sm_count() * per_sm;
  const int most = per_sm > 1 || tiles * 16 <= slots ? 8 : 4;
  int split = 1;
  while (split < most && tiles * split * 2 <= slots && units > (int64_t)split * kDecWarps) split *= 2;
  return split;
}

template <int NT>
int launch_nt(const void* a, int64_t a_stride, const void* b_q, const void* b_sf, const float* alpha, int64_t m, int64_t n, int64_t k,
              void* out, int64_t out_stride, cudaStream_t st) {
  const int split = dec_split(n, k, dec_blocks_per_sm<NT>());
  static SmemOptIn opt_in;
  if (int e = opt_in.ensure(k_gemm_w4a16_decode<NT>, dec_smem_bytes<NT>())) return e;
  const dim3 grid((unsigned)(n / kDecRows * split)), block(32 * kDecWarps);
  const auto *x = (const __nv_bfloat16*)a;
  const auto *q = (const uint8_t*)b_q, *sf = (const uint8_t*)b_sf;
  auto *y = (__nv_bfloat16*)out;
  if (split == 1)
    return (int)launch_chain(k_gemm_w4a16_decode<NT>, grid, block, dec_smem_bytes<NT>(), st, x, a_stride, q, sf, alpha, y, out_stride, (int)m, (int)k, 1);
  return (int)launch_clusters(k_gemm_w4a16_decode<NT>, grid, block, dim3((unsigned)split), dec_smem_bytes<NT>(), st, x, a_stride, q, sf, alpha, y,
                              out_stride, (int)m, (int)k, split);
}

}  // namespace

// Where this kernel is the faster one: up to 16 rows always; up to 32 while a warp takes at most four units of K, in one wave of
// blocks. Its issue time grows with the units and nothing overlaps them, the tile kernel's does not (microseconds a call among
// others, here / tile kernel: 32 x 8192 x 4096, four units, 17.6 / 25.7; 32 x 4096 x 8192, four, 20.1 / 21.9; 32 x 4096 x 12288, six,
// 33.5 / 31.7; 32 x 6144 x 8192, eight, 43.1 / 30.8; 32 x 8192 x 12288, twelve, 69.6 / 54.2; two waves, 32 x 16384 x 4096, 44.5 / 42.6).
// By N and K alone within a range, so a row has one value in all batches of the range.
bool w4a16_decode_wins(int64_t m, int64_t n, int64_t k) {
  if (m <= 16) return true;
  if (m > kW4A16DecodeMaxM) return false;
  const int64_t split = dec_split(n, k, dec_blocks_per_sm<4>()), tiles = n / kDecRows, units = k / kDecUnit, sms = sm_count();
  return tiles * split <= sms && (units + split * kDecWarps - 1) / (split * kDecWarps) <= 4;
}

int launch_gemm_w4a16_decode(const void* a, int64_t a_stride, const void* b_q, const void* b_sf, const float* alpha, int64_t m,
                             int64_t n, int64_t k, void* out, int64_t out_stride, cudaStream_t st) {
  if (m <= 8) return launch_nt<1>(a, a_stride, b_q, b_sf, alpha, m, n, k, out, out_stride, st);
  if (m <= 16) return launch_nt<2>(a, a_stride, b_q, b_sf, alpha, m, n, k, out, out_stride, st);
  return launch_nt<4>(a, a_stride, b_q, b_sf, alpha, m, n, k, out, out_stride, st);
}

}  // namespace b200
