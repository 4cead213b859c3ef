// Internal launch interface shared by the kernel files and the C-ABI layer (api.cu).
#pragma once
#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include <atomic>

namespace b200 {

enum { kGemmDense = 0, kGemmFc1 = 1, kGemmFc2 = 2 };

// True unless the environment says B200MOE_PDL=0 (read once): launches carry the programmatic-stream-serialization
// attribute, so consecutive kernels of the layer overlap launch latency and prologue (see pdl_wait in ptx.cuh).
bool pdl_enabled();

// Multiprocessors of the current device (queried once per device, then cached).
int sm_count();

// cudaFuncAttributeMaxDynamicSharedMemorySize belongs to a (kernel, device) pair: one of these per kernel remembers on
// which devices the opt-in has been made, so that a process driving several GPUs configures each of them.
struct SmemOptIn {
  std::atomic<unsigned long long> done{0};
  template <class Kernel>
  int ensure(Kernel kern, int bytes) {
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return (int)e;
    const unsigned long long bit = 1ull << (dev & 63);
    if (dev < 64 && (done.load(std::memory_order_acquire) & bit)) return 0;
    e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
    if (e != cudaSuccess) return (int)e;
    if (dev < 64) done.fetch_or(bit, std::memory_order_release);
    return 0;
  }
  // which devices have been configured (bit d = device d); for tests of the bookkeeping
  unsigned long long mask() const { return done.load(std::memory_order_acquire); }
};

template <typename... KArgs, typename... Args>
inline cudaError_t launch_chain(void (*kern)(KArgs...), dim3 grid, dim3 block, size_t smem, cudaStream_t st, Args&&... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = pdl_enabled() ? 1 : 0;
  return cudaLaunchKernelEx(&cfg, kern, static_cast<KArgs>(args)...);
}

// The same for a kernel that runs as clusters of more than one block. Such a kernel never calls pdl_trigger: what follows it is released by
// its end alone, so blocks of a next launch that wait on the SMs and clusters that still look for room cannot meet. (A cluster kernel
// and a launch of several waves, both programmatic, once did not finish when called back to back: see gemm_w4a16_expand.cu.)
// A trigger gave nothing: W4A16 of 16 x 4096 x 12288 17.2 us a call with it, 16.8 without; without the attribute 18.4.
template <typename... KArgs, typename... Args>
inline cudaError_t launch_clusters(void (*kern)(KArgs...), dim3 grid, dim3 block, dim3 cluster, size_t smem, cudaStream_t st, Args&&... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = cluster.x;
  attr[0].val.clusterDim.y = cluster.y;
  attr[0].val.clusterDim.z = cluster.z;
  attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[1].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = pdl_enabled() ? 2 : 1;
  return cudaLaunchKernelEx(&cfg, kern, static_cast<KArgs>(args)...);
}

// Device buffers produced by the route-map build.
struct RouteMapBuffers {
  int32_t* block_hist;     // [nblk, E'] scratch
  int32_t* counts;         // [E']
  int32_t* seg_start;      // [E' + 1], multiples of 128
  int32_t* tile_expert;    // [tile_capacity]
  int32_t* tile_row0;      // [tile_capacity]
  int32_t* tile_rows;      // [tile_capacity] valid rows of the tile (1..128)
  int32_t* totals;         // {n_tiles, rows in use (multiple of 128), valid routes, n_pairs}
  int32_t* pair_expert;    // [tile_capacity] 256-row items of the CTA-pair GEMM (may be null: not built)
  int32_t* pair_row0;      // [tile_capacity]
  int32_t* pair_rows;      // [tile_capacity] valid rows of the pair (1..256)
  int32_t* row_of;         // [T, K'] permuted row of a route, -1 when invalid
  int32_t* tok_of_row;     // [row_capacity] token of a permuted row; padding rows (past tile_rows of tile row/128) are unspecified
  float* weight_of_row;    // [row_capacity] routing weight of a permuted row
  int64_t row_capacity;
};

struct GemmParams {
  const int32_t* tile_expert;   // null: dense (expert 0, m-tiles are consecutive 128-row blocks)
  const int32_t* tile_row0;
  const int32_t* tile_rows;
  const int32_t* n_tiles_ptr;   // device count of m-tiles, or null -> n_tiles_static
  int n_tiles_static;
  int M;                        // rows of A (dense mode only)
  int64_t rows_hint;            // most rows of A this launch can hold: picks the form at long k-loops (epilogue width, copier warps),
                                // nothing else; 0 = unknown, as for few
  int N;                        // weight rows per expert (2I for FC1, H for FC2)
  int K;                        // reduction length in FP4 elements
  const int32_t* a_tok;         // FC1 only, non-null: the A map covers the TOKEN rows (box {128, 1}) and row r of a tile is fetched from
                                // token a_tok[row0 + r] by TMA gather; null: the A map covers pre-permuted rows
  const uint8_t* sfa;           // A scales, 128x4 tiles [rows/128][K/64][512]
  const uint8_t* sfb;           // B scales, 128x4 tiles [E*N/128][K/64][512]
  uint8_t* act_q;               // FC1 out: packed activations [rows, I/2]
  uint8_t* act_sf;              // FC1 out: activation scales, 128x4 tiles [rows/128][I/64][512]
  __nv_bfloat16* out;           // FC2 / dense out
  int64_t out_stride;           // elements between output rows
  const int32_t* out_row_index; // FC2 only: output row of permuted row r is out_row_index[r] (null = r itself)
  const float* scale_up;        // per expert multipliers of the FC1 accumulators (null = 1)
  const float* scale_gate;
  const float* alpha;           // per expert activation parameters (null = 1 / 0 / no clamp)
  const float* beta;
  const float* limit;
  int act_type;                 // 3 = SwiGLU form gate*sigmoid(alpha*gate)*(up+beta); 10 = SiTU
  const float* out_scale;       // per expert multiplier of the FC2 accumulator (null = 1)
  float dense_alpha;
  int32_t* status;              // device word; first non-zero code sticks (bounded waits report here)
};

int launch_quantize_nvfp4(const void* x, int64_t rows, int64_t cols, int64_t row_stride, float gs, void* payload, void* scales,
                          int sf_layout, bool clear_tile, cudaStream_t st);   // clear_tile: a tiled image's rows beyond the matrix become 0
int launch_sf_to_tiles(const void* src, int64_t rows, int64_t blocks_per_row, void* dst, cudaStream_t st);
int launch_route_topk(const float* logits, const float* bias, int64_t T, int E, int K, int32_t* ids, float* weights,
                      cudaStream_t st);
int launch_router_logits(const void* x, const void* w, int64_t T, int H, int E, float* logits, cudaStream_t st);
int launch_router_logits_tc(const void* x, const void* w, int64_t T, int H, int E, float* logits, int32_t* status, cudaStream_t st);
// While (token tiles) x (64-expert slices) fit one wave: clusters of blocks split the k-steps and meet in distributed shared
// memory. Returns -1 when the shape does not qualify (the caller then uses launch_router_logits_tc).
int launch_router_logits_ksplit(const void* x, const void* w, int64_t T, int H, int E, float* logits, int32_t* status, cudaStream_t st);
int launch_router_logits_small(const void* x, const void* w, int64_t T, int H, int E, float* logits, cudaStream_t st);   // T <= 16
// Router logits and quantiser of T <= 8 contiguous token rows in one launch (row-major scales, global scale in quantize_fast's range).
int launch_front_small(const void* x, const void* w, int64_t T, int H, int E, float* logits, float gs, void* payload, void* scales,
                       cudaStream_t st);
// seg_len > 0: the T token slots are regions of seg_len consecutive slots and only the first seg_valid[slot / seg_len]
// slots of each region hold a token (the receive buffer of the expert-parallel exchange); the rest count as unrouted.
int launch_route_map(const int32_t* ids, const float* scores, int64_t id_stride, int64_t T, int K, int S, int E, int expert_offset,
                     RouteMapBuffers b, cudaStream_t st, int seg_len = 0, const int32_t* seg_valid = nullptr);
// Route map and permute in ONE launch for batches of at most 16384 routes with row-major token scales (decode sizes):
// `route_gather_fits` says whether a call qualifies.
// With `topk` the expert ids come from router logits inside the launch (`route_gather_topk_fits` says whether a call qualifies);
// `ids` / `scores` are then unused and the selection is also stored to topk->ids / topk->weights.
constexpr int kTopkGatherTokens = 8;
constexpr int kTopkGatherThreads = 256;
// Routes that a block of the one-launch form owns: one row per warp while the SMs last.
inline int route_gather_chunk(int64_t total, int threads, int sms) {
  const int64_t want = (total + threads / 32 - 1) / (threads / 32), blocks = want < sms ? want : sms;
  return (int)((total + blocks - 1) / blocks);
}
// One token per warp, at most 8 experts per lane, and one warp that owns a block's routes: at most 32 of them.
inline bool route_gather_topk_fits(int64_t T, int K, int S, int E, int sms) {
  const int64_t total = T * (K + S);
  return T >= 1 && T <= kTopkGatherTokens && K >= 1 && K <= 32 && E <= 256 && total <= 1024 &&
         route_gather_chunk(total, kTopkGatherThreads, sms) <= 32;
}
struct TopkView {
  const float* logits;
  const float* bias;
  int32_t* ids;
  float* weights;
};
bool route_gather_fits(int64_t T, int K, int S, int E, int H);
int launch_route_gather(const int32_t* ids, const float* scores, int64_t id_stride, int64_t T, int K, int S, int E, int expert_offset,
                        RouteMapBuffers b, const void* hid_q, const void* hid_sf, int64_t q_stride, int64_t sf_stride, int H, void* a_q,
                        void* a_sf, cudaStream_t st, int seg_len = 0, const int32_t* seg_valid = nullptr, const TopkView* topk = nullptr);
int launch_route_map_static(const int32_t* ids, const float* scores, int64_t T, int K, int S, int E, int expert_offset,
                            RouteMapBuffers b, cudaStream_t st);
int launch_ep_visits(const int32_t* ids, int64_t T, int K, int experts_per_rank, int world, int32_t* rank_slots, cudaStream_t st);
int launch_ep_pack(const void* hid_q, const void* hid_sf, const int32_t* ids, const float* weights, const int32_t* tok_of_row,
                   const int32_t* tile_expert, const int32_t* tile_rows, const int32_t* totals, int H, int K, int experts_per_rank,
                   int world, int64_t row_bytes, int64_t row_capacity, void* out, cudaStream_t st);
int launch_gather_rows(const void* hid_q, const void* hid_sf, int hid_sf_tiled, int64_t q_stride, int64_t sf_stride,
                       const int32_t* tok_of_row, const int32_t* tile_rows, const int32_t* totals,
                       int H, int64_t row_capacity, void* a_q, void* a_sf, cudaStream_t st);
int launch_finalize(const void* rout, const int32_t* row_of, const float* weight_of_row, int64_t T, int KK, int H, void* out,
                    int64_t out_stride, cudaStream_t st);
int make_operand_map(CUtensorMap* map, const void* base, uint64_t rows, uint64_t row_bytes, uint32_t box_rows,
                     uint64_t pitch_bytes = 0);   // pitch 0 = rows are contiguous
int launch_gemm_w4a16(const void* a, int64_t a_stride, const void* b_q, const void* b_sf, const float* alpha, int64_t m, int64_t n,
                      int64_t k, void* out, int64_t out_stride, void* workspace, int64_t workspace_bytes, int32_t* status,
                      cudaStream_t st);
// A handful of tokens (gemm_w4a16_decode.cu): no workspace, one launch.
constexpr int kW4A16DecodeMaxM = 32;
bool w4a16_decode_wins(int64_t m, int64_t n, int64_t k);
int launch_gemm_w4a16_decode(const void* a, int64_t a_stride, const void* b_q, const void* b_sf, const float* alpha, int64_t m,
                             int64_t n, int64_t k, void* out, int64_t out_stride, cudaStream_t st);
// Many tokens (gemm_w4a16_expand.cu): the weights expanded to bf16 once, in a scratch of n * k * 2 bytes, then a bf16 GEMM.
constexpr int64_t kW4A16ExpandMax = 1ll << 28;
bool w4a16_expand_wins(int64_t m, int64_t n, int64_t k);
// Width of the tile kernel above 128 rows: narrow tiles while all of them run at once.
inline bool w4a16_wide_tiles(int64_t m, int64_t n, int sms) { return n % 256 == 0 && (m + 255) / 256 * (n / 256) * 2 > sms; }
// A workspace that can hold them. The expansion stores 32 bytes at a time; callers may hand in memory on a 16-byte boundary only, and
// such a call takes the tile kernel (same bits).
inline bool w4a16_expand_room(const void* workspace, int64_t workspace_bytes, int64_t n, int64_t k) {
  return workspace && ((uintptr_t)workspace & 31) == 0 && workspace_bytes >= n * k * 2;
}
int launch_gemm_w4a16_expand(const void* a, int64_t a_stride, const void* b_q, const void* b_sf, const float* alpha, int64_t m,
                             int64_t n, int64_t k, void* out, int64_t out_stride, void* scratch, int32_t* status, cudaStream_t st);
int64_t gemm_w4a16_workspace_bytes(int64_t m, int64_t n, int64_t k);
int make_sf_map(CUtensorMap* map, const void* base, uint64_t n_chunks);

// ---- expert-parallel exchange over peer memory (ep_exchange.cu)
constexpr int kEpMaxRanks = 16;
// int32 fields of a rank's control block, each kEpMaxRanks wide and indexed by the peer that writes it
constexpr int kEpCount = 0;                           // rows the peer sent (its segment, padded to 128)
constexpr int kEpRetBase = kEpMaxRanks;               // first row of that segment in the peer's return buffer
constexpr int kEpFlagDispatch = 2 * kEpMaxRanks;      // step counter: the peer's rows and the two fields above have landed
constexpr int kEpFlagReturn = 3 * kEpMaxRanks;        // step counter: the peer has written its results into my return buffer
constexpr int kEpCtrlInts = 4 * kEpMaxRanks;
struct EpPeers {                   // addresses for the current step's parity, passed to kernels by value
  int32_t world, rank;
  uint8_t* recv[kEpMaxRanks];      // [d]: this rank's region inside rank d's receive buffer
  int32_t* ctrl[kEpMaxRanks];      // [d]: rank d's control block
  void* ret[kEpMaxRanks];          // [s]: rank s's return buffer (bf16 rows)
};
int launch_ep_dispatch(const void* hid_q, const void* hid_sf, const int32_t* ids, const float* weights, const int32_t* tok_of_row,
                       const int32_t* tile_expert, const int32_t* tile_rows, const int32_t* seg_start, const int32_t* totals, int H,
                       int K, int experts_per_rank, int64_t row_bytes, int64_t row_capacity, const EpPeers& peers, int epoch, int64_t T,
                       int shared_slots, int shared_base, int32_t* row_of, float* weight_of_row, unsigned int* done_counter,
                       cudaStream_t st);
int launch_ep_wait(const int32_t* flags, int n, int epoch, int32_t* status, int code, cudaStream_t st);
int launch_ep_post(const EpPeers& peers, int field, int epoch, cudaStream_t st);
int launch_finalize_ep(const void* rout, const int32_t* row_of, const float* weight_of_row, int64_t T, int KK, int H,
                       const EpPeers& peers, const int32_t* ctrl, int seg_len, cudaStream_t st);
int launch_gemm_nvfp4_pair(int mode, const CUtensorMap& ta, const CUtensorMap& tb, const CUtensorMap& tsa, const CUtensorMap& tsb,
                           const GemmParams& p, int n_clusters, cudaStream_t st);
// A-operand maps with 128-, 64- and 16-row boxes (dense and TMA-gathered launches use the first only).
struct ActMaps {
  CUtensorMap rows128, rows64, rows16;
};
int launch_gemm_nvfp4(int mode, int bn, const ActMaps& ta, const CUtensorMap& tb, const GemmParams& p, int grid,
                      cudaStream_t st);

}  // namespace b200
