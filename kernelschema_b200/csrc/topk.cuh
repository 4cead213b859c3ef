// Top-k selection and softmax of one token by one warp (see router.cu for the contract).
#pragma once
#include "kernels.cuh"
#include "ptx.cuh"

namespace b200 {

// fp32 -> unsigned key in the same order; -inf and NaN, which are never selected, become 0 (every other key is larger) and
// both zeros share a key.
DEV uint32_t logit_key(float x) {
  if (!(x > -INFINITY)) return 0u;
  const uint32_t u = __float_as_uint(x + 0.0f);
  return u ^ (u >> 31 ? 0xFFFFFFFFu : 0x80000000u);
}
DEV float key_logit(uint32_t k) { return k ? __uint_as_float(k ^ (k >> 31 ? 0x80000000u : 0xFFFFFFFFu)) : -INFINITY; }

// PL = logits kept per lane (experts <= 32 * PL); the loops are unrolled for the instantiated size only. The K selection rounds
// are a serial chain, so each is two warp-wide reductions (largest key, then lowest expert that has it) instead of five
// exchange steps of (value, index) pairs.
// Lane k < K gets the k-th expert and its weight.
template <int PL>
DEV void topk_token(const float* __restrict__ logits, const float* __restrict__ bias, int E, int K, int lane, int& id, float& weight) {
  uint32_t v[PL];
#pragma unroll
  for (int i = 0; i < PL; ++i) {
    const int e = i * 32 + lane;
    float x = -INFINITY;
    if (e < E) {
      x = logits[e];
      if (bias) x = __fadd_rn(x, bias[e]);
    }
    v[i] = logit_key(x);
  }
  float sel = 0.f;      // lane k keeps the k-th selected logit
  int sel_id = -1;
  uint32_t mine = 0;    // largest key of this lane
#pragma unroll
  for (int i = 0; i < PL; ++i) mine = max(mine, v[i]);
  for (int k = 0; k < K; ++k) {
    const uint32_t best = __reduce_max_sync(0xFFFFFFFFu, mine);
    uint32_t at = 0x7FFFFFFFu;
    if (mine == best && best != 0u) {
#pragma unroll
      for (int i = PL - 1; i >= 0; --i)
        if (v[i] == best) at = (uint32_t)(i * 32 + lane);
    }
    const int best_e = (int)__reduce_min_sync(0xFFFFFFFFu, at);
    if (lane == k) { sel = key_logit(best); sel_id = best_e; }
    if (at == (uint32_t)best_e && best != 0u) {      // the owner takes it out
      mine = 0;
#pragma unroll
      for (int i = 0; i < PL; ++i) {
        if (i * 32 + lane == best_e) v[i] = 0u;
        mine = max(mine, v[i]);
      }
    }
  }
  const float top = __shfl_sync(0xFFFFFFFFu, sel, 0);
  double ex = (lane < K) ? exp((double)sel - (double)top) : 0.0;
  double sum = ex;
#pragma unroll
  for (int off = 16; off > 0; off >>= 1) sum += __shfl_xor_sync(0xFFFFFFFFu, sum, off);
  id = sel_id;
  weight = (float)(ex / sum);
}

}  // namespace b200
