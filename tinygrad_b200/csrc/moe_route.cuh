// The choice of a token's experts, shared by the routing tables (mxfp8.cu) and the one-row expert layer (moe_step.cu).
#pragma once
#include "common.cuh"
#include <math.h>

namespace {

// Choosing a token's experts: one warp per token.  mode 0 (extra/gemm/moe_routing.py:115-116): top-k of the raw logits in
// descending order, weights = softmax over the k.  mode 1 (tinygrad/llm/model.py:118,123-124 with the OLMoE defaults):
// scores = softmax over all experts, top-k listed in ascending order of score, weights = the scores, not renormalised.
// Ties: the lower expert index ranks higher (model.py:35-41).  NaN ranks with -infinity, so that a row of any values has k different choices below n_experts (what
// sorts the pairs indexes by them); a weight is computed from the value itself, NaN included.
constexpr int MAX_E_PER_LANE = 8;   // up to 256 experts; EPL: what a lane has of the number at hand, 1, 2 or 8 (32, 64, 256)

// A value as a number that is greater for what ranks higher; 0: not there, or taken.  (-0 + 0 is 0: the two zeros are equal.)
__device__ __forceinline__ uint32_t rank_key(float v, bool there) {
  const uint32_t u = __float_as_uint((isnan(v) ? -INFINITY : v) + 0.f);
  return there ? u ^ (u >> 31 ? 0xffffffffu : 0x80000000u) : 0;
}
// The expert of the greatest key of a warp, the lowest among equals, is taken: its number, and of `val` what belongs to it.  (Two integer reductions; as five rounds of shuffled
// pairs with the same choices a token's routing took 0.7 us more.)
template <int EPL> __device__ __forceinline__ int take_best(uint32_t (&key)[EPL], const float (&val)[EPL], int lane, float& picked) {
  uint32_t best = 0; unsigned e = 0xffffffffu;
  float v = 0.f;
#pragma unroll
  for (int i = 0; i < EPL; i++) if (key[i] > best) { best = key[i]; v = val[i]; e = i * 32 + lane; }
  const uint32_t top = __reduce_max_sync(0xffffffffu, best);
  e = __reduce_min_sync(0xffffffffu, best == top ? e : 0xffffffffu);
  picked = __shfl_sync(0xffffffffu, v, e & 31);
#pragma unroll
  for (int i = 0; i < EPL; i++) if (i * 32 + lane == (int)e) key[i] = 0;
  return (int)e;
}

// One token by one warp; s_topi (optional): shared memory that gets the choices too.
template <int EPL> __device__ __forceinline__ void route_topk_token(const float* __restrict__ logits, int tok, int n_experts, int k, int mode, int32_t* __restrict__ topi,
                                                 float* __restrict__ weights, int* s_topi) {
  const int lane = threadIdx.x & 31;
  float v[EPL];
  float mx = -INFINITY;
#pragma unroll
  for (int i = 0; i < EPL; i++) {
    const int e = i * 32 + lane;
    v[i] = e < n_experts ? logits[(size_t)tok * n_experts + e] : -INFINITY;
    mx = fmaxf(mx, v[i]);
  }
  mx = warp_max(mx);
  float denom = 0.f;
  if (mode == 1) {
#pragma unroll
    for (int i = 0; i < EPL; i++) denom += (i * 32 + lane < n_experts) ? expf(v[i] - mx) : 0.f;
    denom = warp_sum(denom);
  }
  uint32_t key[EPL];
#pragma unroll
  for (int i = 0; i < EPL; i++) key[i] = rank_key(v[i], i * 32 + lane < n_experts);
  float top1 = 0.f, ksum = 0.f;
#pragma unroll 1
  for (int j = 0; j < k; j++) {
    float bv;
    const int bi = take_best(key, v, lane, bv);
    if (j == 0) top1 = bv;
    const int slot = mode == 1 ? k - 1 - j : j;
    float w;
    if (mode == 1) w = expf(bv - mx) / denom;
    else { w = expf(bv - top1); ksum += w; }
    if (lane == 0) { topi[(size_t)tok * k + slot] = bi; weights[(size_t)tok * k + slot] = w; if (s_topi) s_topi[tok * k + slot] = bi; }
  }
  if (mode == 0) {
    __syncwarp();
    if (lane < k) weights[(size_t)tok * k + lane] /= ksum;
  }
}


// The gating of tinygrad's own MoE block (tinygrad/llm/model.py:110-128), one warp per token:
//   scores = logits (SOFTMAX_WEIGHT) | softmax(logits) | sigmoid(logits) | sqrt(softplus(logits));
//   sel    = the k best of scores (+ sel_bias), listed in ascending order, the lower expert index ranking higher on ties
//            (`pairwise_topk`, model.py:35-41);
//   probs  = scores[sel]; SOFTMAX_WEIGHT: softmax over the k; normalize: / sum; times `scale`.
// The reference's own shortcut is applied by the caller: SOFTMAX with normalize and no bias is run as SOFTMAX_WEIGHT (model.py:116-117).
enum { GATE_SOFTMAX = 1, GATE_SIGMOID = 2, GATE_SOFTMAX_WEIGHT = 3, GATE_SQRT_SOFTPLUS = 4 };     // ExpertGating, model.py:9-13

template <int EPL> __device__ __forceinline__ void route_gating_token(const float* __restrict__ logits, const float* __restrict__ sel_bias, int tok, int n_experts, int k, int gating,
                                                   int normalize, float scale, int32_t* __restrict__ topi, float* __restrict__ weights, int* s_topi) {
  const int lane = threadIdx.x & 31;
  float sc[EPL];
  uint32_t key[EPL];
  float mx = -INFINITY;
#pragma unroll
  for (int i = 0; i < EPL; i++) {
    const int e = i * 32 + lane;
    sc[i] = e < n_experts ? logits[(size_t)tok * n_experts + e] : -INFINITY;
    mx = fmaxf(mx, sc[i]);
  }
  if (gating == GATE_SOFTMAX) {
    mx = warp_max(mx);
    float denom = 0.f;
#pragma unroll
    for (int i = 0; i < EPL; i++) { if (i * 32 + lane < n_experts) { sc[i] = expf(sc[i] - mx); denom += sc[i]; } }
    denom = warp_sum(denom);
#pragma unroll
    for (int i = 0; i < EPL; i++) if (i * 32 + lane < n_experts) sc[i] /= denom;
  } else if (gating == GATE_SIGMOID) {
#pragma unroll
    for (int i = 0; i < EPL; i++) if (i * 32 + lane < n_experts) sc[i] = 1.f / (1.f + expf(-sc[i]));
  } else if (gating == GATE_SQRT_SOFTPLUS) {
#pragma unroll
    for (int i = 0; i < EPL; i++) if (i * 32 + lane < n_experts) sc[i] = sqrtf(sc[i] > 20.f ? sc[i] : log1pf(expf(sc[i])));
  }
#pragma unroll
  for (int i = 0; i < EPL; i++) {
    const int e = i * 32 + lane;
    key[i] = rank_key(sel_bias && e < n_experts ? sc[i] + sel_bias[e] : sc[i], e < n_experts);
  }
  float pv = 0.f;                        // lane j < k keeps the probability of slot j
#pragma unroll 1
  for (int j = 0; j < k; j++) {
    float bs;
    const int bi = take_best(key, sc, lane, bs);
    const int slot = k - 1 - j;          // ascending order of rank
    if (lane == slot) pv = bs;
    if (lane == 0) { topi[(size_t)tok * k + slot] = bi; if (s_topi) s_topi[tok * k + slot] = bi; }
  }
  const bool mine = lane < k;
  if (gating == GATE_SOFTMAX_WEIGHT) {
    const float m2 = warp_max(mine ? pv : -INFINITY);
    const float ev = mine ? expf(pv - m2) : 0.f;
    pv = ev / warp_sum(ev);
  }
  if (normalize) pv = pv / warp_sum(mine ? pv : 0.f);
  if (mine) weights[(size_t)tok * k + lane] = pv * scale;
}

// How a call chooses: gating 0 = `mode` of route_topk_token, else an ExpertGating.
struct RouteRule { int mode, gating, normalize; float scale; const float* sel_bias; };

template <int EPL>
__device__ __forceinline__ void route_token(const RouteRule& r, const float* logits, int tok, int n_experts, int k, int32_t* topi, float* weights, int* s_topi) {
  if (r.gating) route_gating_token<EPL>(logits, r.sel_bias, tok, n_experts, k, r.gating, r.normalize, r.scale, topi, weights, s_topi);
  else route_topk_token<EPL>(logits, tok, n_experts, k, r.mode, topi, weights, s_topi);
}

}  // namespace
