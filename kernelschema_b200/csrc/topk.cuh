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

// Largest of a lane's keys and the lowest expert that has it (a tree: the chain is three comparisons for eight keys).
template <int PL>
DEV void lane_best(const uint32_t (&v)[PL], int lane, uint32_t& key, uint32_t& at) {
  uint32_t k[PL], a[PL];
#pragma unroll
  for (int i = 0; i < PL; ++i) { k[i] = v[i]; a[i] = (uint32_t)(i * 32 + lane); }
#pragma unroll
  for (int w = 1; w < PL; w <<= 1)
#pragma unroll
    for (int i = 0; i + w < PL; i += 2 * w) {
      const bool second = k[i + w] > k[i];
      k[i] = second ? k[i + w] : k[i];
      a[i] = second ? a[i + w] : a[i];
    }
  key = k[0];
  at = a[0];
}

// PL = logits kept per lane (experts <= 32 * PL); the loops are unrolled for the instantiated size only. The K selection rounds
// are a serial chain, so each is two warp-wide reductions (largest key, then lowest expert that has it) instead of five
// exchange steps of (value, index) pairs.
// v[] = this lane's keys (expert i * 32 + lane); lane k < K gets the k-th selected logit and its expert. No branches.
template <int PL>
DEV void topk_select(uint32_t (&v)[PL], int K, int lane, float& sel, int& sel_id) {
  uint32_t mine, mine_at, sel_key = 0x80000000u;      // the key of 0.0f
  sel_id = -1;
  lane_best<PL>(v, lane, mine, mine_at);
  for (int k = 0; k < K; ++k) {
    const uint32_t best = __reduce_max_sync(0xFFFFFFFFu, mine);
    const uint32_t at = __reduce_min_sync(0xFFFFFFFFu, mine == best && best != 0u ? mine_at : 0x7FFFFFFFu);
    sel_key = lane == k ? best : sel_key;
    sel_id = lane == k ? (int)at : sel_id;
#pragma unroll
    for (int i = 0; i < PL; ++i) v[i] = (uint32_t)(i * 32 + lane) == at ? 0u : v[i];
    lane_best<PL>(v, lane, mine, mine_at);
  }
  sel = key_logit(sel_key);
}

template <int PL>
DEV void load_keys(const float* __restrict__ logits, const float* __restrict__ bias, int E, int lane, uint32_t (&v)[PL]) {
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
}

// Softmax over the selected logits in fp64: the first K lanes hold a logit, the largest first.
DEV float softmax_lanes(float sel, int K, int lane) {
  const float top = __shfl_sync(0xFFFFFFFFu, sel, 0);
  double ex = lane < K ? exp((double)sel - (double)top) : 0.0;
  double sum = ex;
#pragma unroll
  for (int off = 16; off > 0; off >>= 1) sum += __shfl_xor_sync(0xFFFFFFFFu, sum, off);
  return (float)(ex / sum);
}

// One token: lane k < K gets the k-th expert and its weight.
template <int PL>
DEV void topk_token(const float* __restrict__ logits, const float* __restrict__ bias, int E, int K, int lane, int& id, float& weight) {
  uint32_t v[PL];
  load_keys<PL>(logits, bias, E, lane, v);
  float sel;
  topk_select<PL>(v, K, lane, sel, id);
  weight = softmax_lanes(sel, K, lane);
}

}  // namespace b200
