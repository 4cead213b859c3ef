// bf16 -> NVFP4 quantiser (16-element blocks, E4M3 block scale, optional fp32 global scale).
//
// Follows, bit for bit, the reference input generator's quantize():
//   moe/nvfp4_fused_moe/problem/input.py:53-71            (global scale 1)
//   gemm/dense/bf16_nvfp4_gemm/problem/input.py:40-64     (global scale != 1)
// One thread owns one 16-element block: 32 bytes loaded, one 64-bit payload store, one scale byte.
// HBM-bound: 2 B read + 0.5625 B written per element.
#include <math.h>

#include "kernels.cuh"
#include "ptx.cuh"
#include "quantize.cuh"

namespace b200 {

// Scale byte position inside the 128x4-tiled layout [rows/128][cols/64][32][16]
// (element (row, blk) at [row/128, blk/4, row%32, 4*((row%128)/32) + blk%4]), the layout tcgen05.cp consumes.
DEV size_t sf_tiled_offset(int64_t row, int64_t blk, int64_t chunks_per_row) {
  return ((size_t)(row >> 7) * chunks_per_row + (size_t)(blk >> 2)) * 512 + (size_t)(row & 31) * 16 + (size_t)((row >> 5) & 3) * 4 +
         (size_t)(blk & 3);
}

// A block of threads = rows_per_block rows x threads_per_row 16-element blocks (one integer division per thread). Bound by HBM
// and, next to it, by issue; what hides both is many warps that are each at another point, so a thread holds one block at a
// time in at most 32 registers (64 warps per SM) and a launch is a few waves of blocks: 8192 x 7168 25.0 us with row-major scales
// (6.0 TB/s), 26.1 tiled. One wave of 28 warps per SM with the loads of two rows each in flight and a table of reciprocals in shared
// memory took 31.0 and 32.5, and a batch of 64 x 7168, which waits for the table, 2.5 against 2.0. Joining four scale bytes by
// shuffles into one store costs more than the stores (27.0).
// WIDE: rows start on 32-byte boundaries, one 256-bit load per block. CLEAR: tiled scales, and the rows that the last tile has beyond the
// matrix become zero (in the launch instead of a memset before it: 3001 x 7168 19.4 -> 15.1 us a call; a form of its own because
// its code costs the others 0.4 us at 8192 x 7168).
template <bool EXACT_DIV, bool WIDE, bool CLEAR>
__global__ void __launch_bounds__(256, EXACT_DIV ? 1 : 8) k_quantize_nvfp4(const __nv_bfloat16* __restrict__ x, int64_t rows, int blocks_per_row,
                                                        int64_t row_stride, float gs, uint8_t* __restrict__ payload,
                                                        uint8_t* __restrict__ scales, int sf_layout, int threads_per_row,
                                                        int rows_per_block) {
  pdl_trigger();
  const float rgs = __frcp_rn(gs);
  const int r = rows_per_block == 1 ? ((int)threadIdx.x >= threads_per_row) : (int)threadIdx.x / threads_per_row;
  const int blk0 = (int)threadIdx.x - r * threads_per_row;
  if (r >= rows_per_block) return;
  pdl_wait();
  for (int64_t row = (int64_t)blockIdx.x * rows_per_block + r; row < rows; row += (int64_t)gridDim.x * rows_per_block)
    for (int blk = blk0; blk < blocks_per_row; blk += threads_per_row) {
      const __nv_bfloat16* src = x + row * row_stride + blk * 16;
      uint32_t w[8];
      if (WIDE) {
        asm volatile("ld.global.nc.v8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
                     : "=r"(w[0]), "=r"(w[1]), "=r"(w[2]), "=r"(w[3]), "=r"(w[4]), "=r"(w[5]), "=r"(w[6]), "=r"(w[7])
                     : "l"(src));
      } else {
        const uint4 lo = __ldg(reinterpret_cast<const uint4*>(src)), hi = __ldg(reinterpret_cast<const uint4*>(src) + 1);
        w[0] = lo.x; w[1] = lo.y; w[2] = lo.z; w[3] = lo.w;
        w[4] = hi.x; w[5] = hi.y; w[6] = hi.z; w[7] = hi.w;
      }
      uint32_t packed[2];
      const uint32_t sbyte = quantize_block<EXACT_DIV>(w, gs, rgs, packed);
      *reinterpret_cast<uint2*>(payload + row * ((int64_t)blocks_per_row * 8) + (int64_t)blk * 8) = make_uint2(packed[0], packed[1]);
      scales[sf_layout == 0 ? (size_t)(row * blocks_per_row + blk) : sf_tiled_offset(row, blk, blocks_per_row >> 2)] = (uint8_t)sbyte;
    }
  if (CLEAR) {                                       // a word at a time
    const int words = blocks_per_row >> 2, pad_words = (int)(-rows & 127) * words, active = rows_per_block * threads_per_row;
    for (int i = (int)blockIdx.x * active + (int)threadIdx.x; i < pad_words; i += (int)gridDim.x * active)
      *reinterpret_cast<uint32_t*>(scales + sf_tiled_offset(rows + i / words, (int64_t)(i % words) * 4, words)) = 0u;
  }
}

// Row-major scale bytes [rows, cols/16] -> 128x4 tiles; rows beyond `rows` up to the next multiple of 128 become 0.
__global__ void k_sf_to_tiles(const uint8_t* __restrict__ src, int64_t rows, int64_t blocks_per_row, uint8_t* __restrict__ dst) {
  const int64_t rows_pad = (rows + 127) & ~(int64_t)127;
  const int64_t words_per_row = blocks_per_row >> 2;
  const int64_t total = rows_pad * words_per_row;
  for (int64_t idx = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; idx < total; idx += (int64_t)gridDim.x * blockDim.x) {
    const int64_t row = idx / words_per_row;
    const int64_t wd = idx - row * words_per_row;
    uint32_t val = 0;
    if (row < rows) val = *reinterpret_cast<const uint32_t*>(src + row * blocks_per_row + wd * 4);
    *reinterpret_cast<uint32_t*>(dst + sf_tiled_offset(row, wd * 4, words_per_row)) = val;
  }
}

int launch_quantize_nvfp4(const void* x, int64_t rows, int64_t cols, int64_t row_stride, float gs, void* payload, void* scales,
                          int sf_layout, bool clear_tile, cudaStream_t st) {
  if (rows == 0) return 0;
  const int bpr = (int)(cols >> 4);
  // threads of a row: its 16-element blocks in equal passes of at most 256; short rows share a block (16384 x 512: 6.0 us, 8.4 with
  // a block per row)
  const int passes = (bpr + 255) / 256;
  const int tpr = (bpr + passes - 1) / passes;
  const int64_t spread = rows / sm_count();                              // a short batch: first a block for every SM
  const int rpb = (int)(spread < 1 ? 1 : spread < 256 / tpr ? spread : 256 / tpr);
  const int threads = (rpb * tpr + 31) / 32 * 32;
  const int64_t most = (int64_t)sm_count() * 32;
  const int64_t want = (rows + rpb - 1) / rpb;
  const int64_t blocks = want < most ? want : most;
  const bool wide = ((uintptr_t)x & 31) == 0 && row_stride % 16 == 0;
  const bool clear = clear_tile && sf_layout != 0 && rows % 128 != 0;
  auto go = [&](auto kern) {
    return (int)launch_chain(kern, dim3((unsigned)blocks), dim3(threads), 0, st, (const __nv_bfloat16*)x, rows, bpr, row_stride, gs,
                             (uint8_t*)payload, (uint8_t*)scales, sf_layout, tpr, rpb);
  };
  if (!quantize_fast(gs)) return clear ? go(k_quantize_nvfp4<true, false, true>) : go(k_quantize_nvfp4<true, false, false>);
  if (wide) return clear ? go(k_quantize_nvfp4<false, true, true>) : go(k_quantize_nvfp4<false, true, false>);
  return clear ? go(k_quantize_nvfp4<false, false, true>) : go(k_quantize_nvfp4<false, false, false>);
}

int launch_sf_to_tiles(const void* src, int64_t rows, int64_t blocks_per_row, void* dst, cudaStream_t st) {
  const int64_t rows_pad = (rows + 127) & ~(int64_t)127;
  const int64_t total = rows_pad * (blocks_per_row >> 2);
  if (total == 0) return 0;
  int64_t blocks = (total + 255) / 256;
  if (blocks > (int64_t)sm_count() * 16) blocks = (int64_t)sm_count() * 16;
  k_sf_to_tiles<<<(unsigned)blocks, 256, 0, st>>>((const uint8_t*)src, rows, blocks_per_row, (uint8_t*)dst);
  return (int)cudaGetLastError();
}

}  // namespace b200
