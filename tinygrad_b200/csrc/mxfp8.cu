// MXFP8 (E4M3 values + one E8M0 scale per 32 along K) mixture-of-experts path:
// activation quantiser, top-k routing tables, row dispatch / combine, SwiGLU + requantise.
// The grouped expert GEMM is in mxfp8_gemm.cu.
//
// Semantics follow extra/gemm/cdna_asm_gemm.py:149-173 (quantize_mxfp8, _mx_block_scale),
// tinygrad/dtype.py:237-260 (E4M3 round-to-nearest-even, saturating), extra/gemm/moe_routing.py:89-131
// (route / dispatch / combine, groups padded to 256 rows) and tinygrad/llm/model.py:35-41,110-130
// (softmax-over-all-experts gating with compare-count top-k, the OLMoE default).
#include "common.cuh"
#include "mxq.cuh"
#include "moe_route.cuh"
#include <cuda_bf16.h>
#include <cuda_fp8.h>
#include <math.h>

namespace {

constexpr int BLOCK_ROW = 256;   // extra/gemm/moe_routing.py:4

__device__ __forceinline__ void bf16x8_to_f32(const uint4& u, float (&v)[8]) {
  const uint32_t w[4] = {u.x, u.y, u.z, u.w};
#pragma unroll
  for (int i = 0; i < 4; i++) { v[2 * i] = __uint_as_float(w[i] << 16); v[2 * i + 1] = __uint_as_float(w[i] & 0xFFFF0000u); }
}
template <typename T> __device__ __forceinline__ void load8(const T* p, float (&v)[8]);
template <> __device__ __forceinline__ void load8<float>(const float* p, float (&v)[8]) {
  const float4 a = *reinterpret_cast<const float4*>(p), b = *reinterpret_cast<const float4*>(p + 4);
  v[0] = a.x; v[1] = a.y; v[2] = a.z; v[3] = a.w; v[4] = b.x; v[5] = b.y; v[6] = b.z; v[7] = b.w;
}
template <> __device__ __forceinline__ void load8<__nv_bfloat16>(const __nv_bfloat16* p, float (&v)[8]) {
  bf16x8_to_f32(*reinterpret_cast<const uint4*>(p), v);
}
__device__ __forceinline__ float amax8_quad(const float (&v)[8]) {      // |max| over the 32 values held by 4 neighbouring lanes
  float m = 0.f;
#pragma unroll
  for (int i = 0; i < 8; i++) m = fmaxf(m, fabsf(v[i]));
  m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, 1));
  return fmaxf(m, __shfl_xor_sync(0xffffffffu, m, 2));
}

// One warp per 256 consecutive values of a row: 4 lanes share a block of 32, a lane holds 8 values (16-byte loads, 8-byte stores).
// Rows of x go to rows dest[r] of the outputs (dest == nullptr: identity); `fan` consecutive dest entries per input row.
template <typename T>
__global__ void quantize_mxfp8_kernel(const T* __restrict__ x, int64_t rows, int k, const int32_t* __restrict__ dest, int fan,
                                      uint8_t* __restrict__ q, uint8_t* __restrict__ e8) {
  pdl_launch_dependents();
  pdl_wait();
  const int lane = threadIdx.x & 31;
  const int64_t warp = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int kb = k >> 5, chunks = (kb + 7) >> 3;
  if (warp >= rows * chunks) return;
  const int64_t r = warp / chunks;
  const int b = (int)(warp - r * chunks) * 8 + (lane >> 2), col = b * 32 + (lane & 3) * 8;
  const bool valid = b < kb;
  float v[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
  if (valid) load8<T>(x + r * k + col, v);
  const uint8_t e = mx_scale_exponent(amax8_quad(v));
  const uint2 pk = mx_quant8(v, e);
  if (!valid) return;
  for (int f = 0; f < fan; f++) {
    const int64_t o = dest ? (int64_t)dest[r * fan + f] : r;
    if (o < 0) continue;
    *reinterpret_cast<uint2*>(q + o * k + col) = pk;
    if ((lane & 3) == 0) e8[o * kb + b] = e;
  }
}

// SwiGLU between the two expert GEMMs: h = [gate | up] (bf16, [m, 2f]) -> act = silu(gate) * up computed in fp32,
// rounded to bf16 as a tensor would be stored, then quantised like any activation.  Same work split as the quantiser.
__global__ void swiglu_quant_kernel(const __nv_bfloat16* __restrict__ h, int64_t rows, const int32_t* __restrict__ rows_used, int f,
                                    uint8_t* __restrict__ q, uint8_t* __restrict__ e8) {
  pdl_launch_dependents();
  pdl_wait();
  const int lane = threadIdx.x & 31;
  const int64_t warp = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int kb = f >> 5, chunks = (kb + 7) >> 3;
  if (rows_used) rows = min(rows, (int64_t)*rows_used);
  if (warp >= rows * chunks) return;
  const int64_t r = warp / chunks;
  const int b = (int)(warp - r * chunks) * 8 + (lane >> 2), col = b * 32 + (lane & 3) * 8;
  const bool valid = b < kb;
  float v[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
  if (valid) {
    float g[8], u[8];
    load8<__nv_bfloat16>(h + r * 2 * f + col, g);
    load8<__nv_bfloat16>(h + r * 2 * f + f + col, u);
#pragma unroll
    for (int i = 0; i < 8; i++) v[i] = __bfloat162float(__float2bfloat16_rn((g[i] / (1.f + expf(-g[i]))) * u[i]));
  }
  const uint8_t e = mx_scale_exponent(amax8_quad(v));
  const uint2 pk = mx_quant8(v, e);
  if (!valid) return;
  *reinterpret_cast<uint2*>(q + r * f + col) = pk;
  if ((lane & 3) == 0) e8[r * kb + b] = e;
}

template <int EPL>
__global__ void route_choose_kernel(const RouteRule r, const float* __restrict__ logits, int n_tokens, int n_experts, int k, int32_t* __restrict__ topi,
                                    float* __restrict__ weights) {
  pdl_launch_dependents();
  pdl_wait();
  const int tok = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  if (tok < n_tokens) route_token<EPL>(r, logits, tok, n_experts, k, topi, weights, nullptr);
}

// routing, steps 2-4: stable counting sort of the T*k (token, slot) pairs by expert.
// dest_row[i] = off[e_i] + (number of pairs before i with the same expert); off = cumulative group sizes padded to 256.
constexpr int ROUTE_CHUNK = 1024;
// A choice made by the caller that is no expert has no row: dest_row -1, which the kernels that move rows pass over.
__device__ __forceinline__ int known_expert(int e, int n_experts) { return e >= 0 && e < n_experts ? e : -1; }
// ends (optional) [n_experts]: off + size, the row behind each expert's last.

// Padded offsets from the group sizes `tot` (shared memory), by one warp.
__device__ __forceinline__ void route_offsets(const int* tot, int n_experts, int pad, int32_t* __restrict__ off, int32_t* __restrict__ counts, int32_t* __restrict__ ends,
                                              int* s_off) {
  const int lane = threadIdx.x & 31;
  int carry = 0;
#pragma unroll 1
  for (int e0 = 0; e0 < n_experts; e0 += 32) {
    const int e = e0 + lane, n = e < n_experts ? tot[e] : 0, padded = (n + pad - 1) / pad * pad;
    int incl = padded;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) { const int v = __shfl_up_sync(0xffffffffu, incl, o); if (lane >= o) incl += v; }
    const int at = carry + incl - padded;
    if (e < n_experts) {
      off[e + 1] = at + padded;
      if (counts) counts[e] = n;
      if (ends) ends[e] = at + n;
      if (s_off) s_off[e] = at;
    }
    carry += __shfl_sync(0xffffffffu, incl, 31);
  }
  if (lane == 0) off[0] = 0;
}

// The whole routing of at most ROUTE_CHUNK pairs and ROUTE_ONE_TOKENS tokens in one CTA: a warp per token, then the counting sort in shared memory.
// As four launches it took 18.5 us whatever the size, nearly all of it launches.  logits == nullptr: the choices are there already (topi); more tokens than warps are
// chosen for by a kernel of their own in front: 256 tokens x 4 took 34.5 us as eight tokens a warp here, 5.1 so; 64 x 2 6.9, 3.7.
constexpr int ROUTE_ONE_TOKENS = 32;
template <int EPL>
__global__ void __launch_bounds__(ROUTE_CHUNK) route_one_kernel(const RouteRule r, const float* __restrict__ logits, int n_tokens, int n_experts, int k, int pad,
                                                                int32_t* __restrict__ topi, float* __restrict__ weights, int32_t* __restrict__ dest_row,
                                                                int32_t* __restrict__ off, int32_t* __restrict__ counts, int32_t* __restrict__ ends) {
  extern __shared__ int s_route[];                // [ROUTE_CHUNK choices][n_experts sizes][n_experts offsets][warps][n_experts]
  int *s_topi = s_route, *s_tot = s_topi + ROUTE_CHUNK, *s_off = s_tot + n_experts, *s_wcnt = s_off + n_experts;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, n = n_tokens * k, n_warps = (n + 31) >> 5;
  for (int i = threadIdx.x; i < n_warps * n_experts; i += ROUTE_CHUNK) s_wcnt[i] = 0;
  pdl_launch_dependents();
  pdl_wait();
  if (logits) {
#pragma unroll 1
    for (int tok = warp; tok < n_tokens; tok += ROUTE_CHUNK / 32) route_token<EPL>(r, logits, tok, n_experts, k, topi, weights, s_topi);
  } else for (int i = threadIdx.x; i < n; i += ROUTE_CHUNK) s_topi[i] = topi[i];
  __syncthreads();
  const int i = threadIdx.x, e = i < n ? known_expert(s_topi[i], n_experts) : -1;
  const unsigned same = __match_any_sync(0xffffffffu, e);
  const int before_in_warp = __popc(same & ((1u << lane) - 1));
  if (e >= 0 && before_in_warp == 0) s_wcnt[warp * n_experts + e] = __popc(same);
  __syncthreads();
  for (int x = threadIdx.x; x < n_experts; x += ROUTE_CHUNK) {
    int run = 0;
    for (int w = 0; w < n_warps; w++) { const int v = s_wcnt[w * n_experts + x]; s_wcnt[w * n_experts + x] = run; run += v; }
    s_tot[x] = run;
  }
  __syncthreads();
  if (warp == 0) route_offsets(s_tot, n_experts, pad, off, counts, ends, s_off);
  __syncthreads();
  if (i < n) dest_row[i] = e >= 0 ? s_off[e] + s_wcnt[warp * n_experts + e] + before_in_warp : -1;
}

__global__ void __launch_bounds__(ROUTE_CHUNK) route_count_kernel(const int32_t* __restrict__ topi, int n, int n_experts, int32_t* __restrict__ counts) {
  extern __shared__ int s_cnt[];
  pdl_launch_dependents();
  pdl_wait();
  for (int e = threadIdx.x; e < n_experts; e += blockDim.x) s_cnt[e] = 0;
  __syncthreads();
  const int i = blockIdx.x * ROUTE_CHUNK + threadIdx.x;
  const int e = i < n ? known_expert(topi[i], n_experts) : -1;
  if (e >= 0) atomicAdd(&s_cnt[e], 1);      // integer counts: the order of the adds does not matter
  __syncthreads();
  for (int x = threadIdx.x; x < n_experts; x += blockDim.x) counts[(size_t)blockIdx.x * n_experts + x] = s_cnt[x];
}

// one warp per expert: exclusive scan of its chunk counts (in place, 32 chunks at a time); then one warp builds the padded offsets
__global__ void __launch_bounds__(ROUTE_CHUNK) route_scan_kernel(int32_t* __restrict__ counts, int n_chunks, int n_experts, int32_t* __restrict__ off, int pad,
                                                                 int32_t* __restrict__ counts_out, int32_t* __restrict__ ends) {
  extern __shared__ int s_tot[];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  pdl_launch_dependents();
  pdl_wait();
#pragma unroll 1
  for (int e = warp; e < n_experts; e += ROUTE_CHUNK / 32) {
    int run = 0;
#pragma unroll 1
    for (int c0 = 0; c0 < n_chunks; c0 += 32) {
      const int c = c0 + lane, v = c < n_chunks ? counts[(size_t)c * n_experts + e] : 0;
      int incl = v;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) { const int u = __shfl_up_sync(0xffffffffu, incl, o); if (lane >= o) incl += u; }
      if (c < n_chunks) counts[(size_t)c * n_experts + e] = run + incl - v;
      run += __shfl_sync(0xffffffffu, incl, 31);
    }
    if (lane == 0) s_tot[e] = run;
  }
  __syncthreads();
  if (warp == 0) route_offsets(s_tot, n_experts, pad, off, counts_out, ends, nullptr);
}

// rows of `row_bytes` bytes moved by an index table: scatter dst[idx[i]] = src[i] or gather dst[i] = src[idx[i]]; idx < 0 skips
template <typename V>
__global__ void permute_rows_kernel(const V* __restrict__ src, const int32_t* __restrict__ idx, int64_t n_rows, int row_vecs, V* __restrict__ dst,
                                    int gather) {
  const int64_t r = blockIdx.x;
  const int j = idx[r];
  if (j < 0) return;
  const V* s = src + (gather ? (int64_t)j : r) * row_vecs;
  V* d = dst + (gather ? r : (int64_t)j) * row_vecs;
  for (int i = threadIdx.x; i < row_vecs; i += blockDim.x) d[i] = s[i];
}

__global__ void __launch_bounds__(ROUTE_CHUNK) route_place_kernel(const int32_t* __restrict__ topi, int n, int n_experts,
                                                                  const int32_t* __restrict__ counts, const int32_t* __restrict__ off,
                                                                  int32_t* __restrict__ dest_row) {
  extern __shared__ int s_wcnt[];                 // [32 warps][n_experts] pairs of each expert seen by each warp
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  for (int j = threadIdx.x; j < 32 * n_experts; j += blockDim.x) s_wcnt[j] = 0;
  pdl_launch_dependents();
  pdl_wait();
  __syncthreads();
  const int i = blockIdx.x * ROUTE_CHUNK + threadIdx.x;
  const int e = i < n ? known_expert(topi[i], n_experts) : -1;
  const unsigned same = __match_any_sync(0xffffffffu, e);
  const int before_in_warp = __popc(same & ((1u << lane) - 1));
  if (e >= 0 && before_in_warp == 0) s_wcnt[warp * n_experts + e] = __popc(same);
  __syncthreads();
  if (e >= 0) {
    int before = counts[(size_t)blockIdx.x * n_experts + e] + before_in_warp;
    for (int w = 0; w < warp; w++) before += s_wcnt[w * n_experts + e];
    dest_row[i] = off[e] + before;
  } else if (i < n) dest_row[i] = -1;
}

// combine (extra/gemm/moe_routing.py:128-131): out[t] = sum_j weights[t, j] * y[dest_row[t*k + j]], fp32 sum in slot order, bf16 out; add_to
// (optional, fp32 [n_tokens, d]): the rounded sum is added to it as well (the residual behind the expert layer)
__device__ __forceinline__ void combine_token(int t, const __nv_bfloat16* __restrict__ y, const int32_t* __restrict__ dest_row, const float* __restrict__ weights, int k, int d,
                                              __nv_bfloat16* __restrict__ out, float* __restrict__ add_to) {
  for (int c = threadIdx.x; c < d; c += blockDim.x) {
    float acc = 0.f;
    for (int j = 0; j < k; j++) {
      const int row = dest_row[(size_t)t * k + j];
      if (row >= 0) acc += weights[(size_t)t * k + j] * __bfloat162float(y[(size_t)row * d + c]);
    }
    const __nv_bfloat16 r = __float2bfloat16_rn(acc);
    out[(size_t)t * d + c] = r;
    if (add_to) add_to[(size_t)t * d + c] += __bfloat162float(r);
  }
}
__global__ void combine_kernel(const __nv_bfloat16* __restrict__ y, const int32_t* __restrict__ dest_row, const float* __restrict__ weights,
                               int n_tokens, int k, int d, __nv_bfloat16* __restrict__ out, float* __restrict__ add_to) {
  pdl_launch_dependents();
  pdl_wait();
  combine_token(blockIdx.x, y, dest_row, weights, k, d, out, add_to);
}
// d % 8 == 0: a thread sums 8 neighbouring columns over the k rows (16-byte loads), same order of additions.  A CTA stages its token's rows and
// weights, so that four rows are in flight at once (4096 tokens x 8 rows of 2048: 34.9 us with the row numbers loaded one by one).  A token with a choice that has no
// row goes the other way as a whole (asked at every load: 28.9 us, 28.5 so).
constexpr int COMBINE_MAX_K = 32;
__global__ void __launch_bounds__(256) combine8_kernel(const __nv_bfloat16* __restrict__ y, const int32_t* __restrict__ dest_row, const float* __restrict__ weights,
                                                       int n_tokens, int k, int d, __nv_bfloat16* __restrict__ out, float* __restrict__ add_to) {
  __shared__ int s_row[COMBINE_MAX_K];
  __shared__ float s_w[COMBINE_MAX_K];
  const int t = blockIdx.x;
  pdl_launch_dependents();
  pdl_wait();
  int row = 0;
  if (threadIdx.x < k) { s_row[threadIdx.x] = row = dest_row[(size_t)t * k + threadIdx.x]; s_w[threadIdx.x] = weights[(size_t)t * k + threadIdx.x]; }
  if (__syncthreads_or(row < 0)) { combine_token(t, y, dest_row, weights, k, d, out, add_to); return; }
  for (int c = threadIdx.x * 8; c < d; c += blockDim.x * 8) {
    float acc[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
    for (int j0 = 0; j0 < k; j0 += 4) {
      uint4 u[4];
#pragma unroll
      for (int j = 0; j < 4; j++) if (j0 + j < k) u[j] = *reinterpret_cast<const uint4*>(y + (size_t)s_row[j0 + j] * d + c);
#pragma unroll
      for (int j = 0; j < 4; j++) {
        if (j0 + j < k) {
          const float w = s_w[j0 + j];
          float v[8];
          bf16x8_to_f32(u[j], v);
#pragma unroll
          for (int i = 0; i < 8; i++) acc[i] += w * v[i];
        }
      }
    }
    uint4 pk;
    __nv_bfloat162* hp = reinterpret_cast<__nv_bfloat162*>(&pk);
#pragma unroll
    for (int i = 0; i < 4; i++) hp[i] = __floats2bfloat162_rn(acc[2 * i], acc[2 * i + 1]);
    *reinterpret_cast<uint4*>(out + (size_t)t * d + c) = pk;
    if (add_to) {
      float v[8];
      bf16x8_to_f32(pk, v);
      float4* x = reinterpret_cast<float4*>(add_to + (size_t)t * d + c);
      float4 a = x[0], b = x[1];
      a.x += v[0]; a.y += v[1]; a.z += v[2]; a.w += v[3]; b.x += v[4]; b.y += v[5]; b.z += v[6]; b.w += v[7];
      x[0] = a; x[1] = b;
    }
  }
}

// ---- launches; pdl: programmatic, behind a kernel of this library on the same stream ----
int quantize_launch(const void* x, int x_dtype, int64_t rows, int k, const int32_t* dest_row, int fan, void* q, void* e8, cudaStream_t st, bool pdl) {
  if (rows < 0 || k <= 0 || (rows && (!x || !q || !e8))) return B200Q_ERR_BAD_ARG;
  if (x_dtype != B200Q_F32 && x_dtype != B200Q_BF16) return B200Q_ERR_BAD_ARG;
  if (k % 32) return B200Q_ERR_BAD_SHAPE;
  if (dest_row ? fan <= 0 : fan != 1) return B200Q_ERR_BAD_ARG;
  if (rows == 0) return B200Q_OK;
  if (((uintptr_t)x | (uintptr_t)q) & 15) return B200Q_ERR_MISALIGNED;
  const int64_t warps = rows * ((k / 32 + 7) / 8);
  const dim3 grid((unsigned)((warps + 7) / 8));
  if (x_dtype == B200Q_F32)
    B200Q_CHECK_CUDA(launch_k(quantize_mxfp8_kernel<float>, grid, dim3(256), 0, st, pdl, (const float*)x, rows, k, dest_row, fan, (uint8_t*)q, (uint8_t*)e8));
  else
    B200Q_CHECK_CUDA(launch_k(quantize_mxfp8_kernel<__nv_bfloat16>, grid, dim3(256), 0, st, pdl, (const __nv_bfloat16*)x, rows, k, dest_row, fan, (uint8_t*)q, (uint8_t*)e8));
  return B200Q_OK;
}

int combine_launch(const void* y_bf16, const int32_t* dest_row, const float* weights, int n_tokens, int k, int d, void* out_bf16, float* add_to, cudaStream_t st,
                   bool pdl) {
  if (!y_bf16 || !dest_row || !weights || !out_bf16 || n_tokens <= 0 || k <= 0 || d <= 0) return B200Q_ERR_BAD_ARG;
  const bool wide = d % 8 == 0 && k <= COMBINE_MAX_K && !(((uintptr_t)y_bf16 | (uintptr_t)out_bf16 | (uintptr_t)add_to) & 15);
  B200Q_CHECK_CUDA(launch_k(wide ? combine8_kernel : combine_kernel, dim3(n_tokens), dim3(256), 0, st, pdl, (const __nv_bfloat16*)y_bf16, dest_row, weights, n_tokens, k, d,
                            (__nv_bfloat16*)out_bf16, add_to));
  return B200Q_OK;
}

// logits == nullptr: the choices are in topi already.
int route_launch(const RouteRule& r, const float* logits, int n_tokens, int n_experts, int k, int pad, int32_t* topi, float* weights, int32_t* dest_row, int32_t* off,
                 int32_t* counts, int32_t* ends, void* scratch, cudaStream_t st, bool pdl) {
  const int n = n_tokens * k, n_chunks = ceil_div(n, ROUTE_CHUNK);
  const bool one = n <= ROUTE_CHUNK;
  if (logits && !(one && n_tokens <= ROUTE_ONE_TOKENS)) {
    auto choose = n_experts <= 32 ? route_choose_kernel<1> : n_experts <= 64 ? route_choose_kernel<2> : route_choose_kernel<MAX_E_PER_LANE>;
    B200Q_CHECK_CUDA(launch_k(choose, dim3(ceil_div(n_tokens, 8)), dim3(256), 0, st, pdl, r, logits, n_tokens, n_experts, k, topi, weights));
    pdl = true;
    logits = nullptr;
  }
  if (one) {
    const size_t smem = (ROUTE_CHUNK + (2 + (size_t)ceil_div(n, 32)) * n_experts) * sizeof(int);      // at most 38 KB
    auto sort = n_experts <= 32 ? route_one_kernel<1> : n_experts <= 64 ? route_one_kernel<2> : route_one_kernel<MAX_E_PER_LANE>;
    B200Q_CHECK_CUDA(launch_k(sort, dim3(1), dim3(ROUTE_CHUNK), smem, st, pdl, r, logits, n_tokens, n_experts, k, pad, topi, weights, dest_row, off, counts, ends));
    return B200Q_OK;
  }
  int32_t* cnt = (int32_t*)scratch;
  B200Q_CHECK_CUDA(launch_k(route_count_kernel, dim3(n_chunks), dim3(ROUTE_CHUNK), n_experts * sizeof(int), st, pdl, topi, n, n_experts, cnt));
  B200Q_CHECK_CUDA(launch_k(route_scan_kernel, dim3(1), dim3(ROUTE_CHUNK), n_experts * sizeof(int), st, true, cnt, n_chunks, n_experts, off, pad, counts, ends));
  B200Q_CHECK_CUDA(launch_k(route_place_kernel, dim3(n_chunks), dim3(ROUTE_CHUNK), 32 * n_experts * sizeof(int), st, true, topi, n, n_experts, cnt, off, dest_row));
  return B200Q_OK;
}

}  // namespace

extern "C" int b200q_quantize_mxfp8(const void* x, int x_dtype, int64_t rows, int k, const int32_t* dest_row, int fan, void* q, void* e8, void* stream) {
  return quantize_launch(x, x_dtype, rows, k, dest_row, fan, q, e8, (cudaStream_t)stream, false);
}

extern "C" int b200q_swiglu_quantize_mxfp8(const void* h_bf16, int64_t rows, const int32_t* rows_used, int f, void* q, void* e8, void* stream) {
  if (rows < 0 || f <= 0 || (rows && (!h_bf16 || !q || !e8))) return B200Q_ERR_BAD_ARG;
  if (f % 32) return B200Q_ERR_BAD_SHAPE;
  if (((uintptr_t)h_bf16 | (uintptr_t)q) & 15) return B200Q_ERR_MISALIGNED;
  if (rows == 0) return B200Q_OK;
  const int64_t warps = rows * ((f / 32 + 7) / 8);
  swiglu_quant_kernel<<<(unsigned)((warps + 7) / 8), 256, 0, (cudaStream_t)stream>>>((const __nv_bfloat16*)h_bf16, rows, rows_used, f, (uint8_t*)q,
                                                                                       (uint8_t*)e8);
  B200Q_CHECK_CUDA(cudaGetLastError());
  return B200Q_OK;
}

extern "C" size_t b200q_moe_route_scratch_bytes(int n_tokens, int n_experts, int k) {
  if (n_tokens <= 0 || n_experts <= 0 || k <= 0) return 0;
  return (size_t)ceil_div(n_tokens * k, ROUTE_CHUNK) * n_experts * sizeof(int32_t);
}

extern "C" int b200q_moe_rows_max(int n_tokens, int n_experts, int k) {   // m_max_for, extra/gemm/moe_routing.py:89-90
  return (ceil_div(n_tokens * k, BLOCK_ROW) + n_experts) * BLOCK_ROW;
}

extern "C" int b200q_moe_route(const float* logits, int n_tokens, int n_experts, int k, int mode, int32_t* topi, float* weights, int32_t* dest_row,
                               int32_t* off, void* scratch, void* stream) {
  return b200q_moe_route_pad(logits, n_tokens, n_experts, k, mode, BLOCK_ROW, topi, weights, dest_row, off, nullptr, scratch, stream);
}

extern "C" int b200q_permute_rows(const void* src, const int32_t* idx, int64_t n_rows, int row_bytes, void* dst, int gather, void* stream) {
  if (n_rows < 0 || row_bytes <= 0 || (n_rows && (!src || !idx || !dst))) return B200Q_ERR_BAD_ARG;
  if (row_bytes % 4) return B200Q_ERR_BAD_SHAPE;
  if (n_rows == 0) return B200Q_OK;
  if (row_bytes % 16 == 0 && !(((uintptr_t)src | (uintptr_t)dst) & 15))
    permute_rows_kernel<uint4><<<(unsigned)n_rows, 128, 0, (cudaStream_t)stream>>>((const uint4*)src, idx, n_rows, row_bytes / 16, (uint4*)dst, gather);
  else
    permute_rows_kernel<uint32_t><<<(unsigned)n_rows, 128, 0, (cudaStream_t)stream>>>((const uint32_t*)src, idx, n_rows, row_bytes / 4, (uint32_t*)dst, gather);
  B200Q_CHECK_CUDA(cudaGetLastError());
  return B200Q_OK;
}

extern "C" int b200q_moe_route_pad(const float* logits, int n_tokens, int n_experts, int k, int mode, int pad, int32_t* topi, float* weights,
                                   int32_t* dest_row, int32_t* off, int32_t* counts, void* scratch, void* stream) {
  if (!logits || !topi || !weights || !dest_row || !off || !scratch || pad <= 0) return B200Q_ERR_BAD_ARG;
  if (n_tokens <= 0 || n_experts <= 0 || k <= 0 || k > n_experts || (mode != 0 && mode != 1)) return B200Q_ERR_BAD_ARG;
  if (n_experts > 32 * MAX_E_PER_LANE || k > 32) return B200Q_ERR_BAD_SHAPE;
  return route_launch(RouteRule{mode, 0, 0, 1.f, nullptr}, logits, n_tokens, n_experts, k, pad, topi, weights, dest_row, off, counts, nullptr, scratch, (cudaStream_t)stream, false);
}

extern "C" int b200q_moe_route_tables(const int32_t* topi, int n_tokens, int n_experts, int k, int pad, int32_t* dest_row, int32_t* off, int32_t* counts,
                                      void* scratch, void* stream) {
  if (!topi || !dest_row || !off || !scratch || pad <= 0 || n_tokens <= 0 || n_experts <= 0 || k <= 0) return B200Q_ERR_BAD_ARG;
  if (n_experts > 32 * MAX_E_PER_LANE) return B200Q_ERR_BAD_SHAPE;
  return route_launch(RouteRule{}, nullptr, n_tokens, n_experts, k, pad, const_cast<int32_t*>(topi), nullptr, dest_row, off, counts, nullptr, scratch, (cudaStream_t)stream, false);
}

extern "C" int b200q_moe_route_gating(const float* logits, const float* sel_bias, int n_tokens, int n_experts, int k, int gating, int normalize, float scale,
                                      int pad, int32_t* topi, float* weights, int32_t* dest_row, int32_t* off, int32_t* counts, void* scratch, void* stream) {
  if (!logits || !topi || !weights || !dest_row || !off || !scratch || pad <= 0) return B200Q_ERR_BAD_ARG;
  if (n_tokens <= 0 || n_experts <= 0 || k <= 0 || k > n_experts || gating < GATE_SOFTMAX || gating > GATE_SQRT_SOFTPLUS) return B200Q_ERR_BAD_ARG;
  if (n_experts > 32 * MAX_E_PER_LANE || k > 32) return B200Q_ERR_BAD_SHAPE;
  return route_launch(RouteRule{0, gating, normalize, scale, sel_bias}, logits, n_tokens, n_experts, k, pad, topi, weights, dest_row, off, counts, nullptr, scratch,
                      (cudaStream_t)stream, false);
}

extern "C" int b200q_moe_combine(const void* y_bf16, const int32_t* dest_row, const float* weights, int n_tokens, int k, int d, void* out_bf16,
                                 void* stream) {
  return combine_launch(y_bf16, dest_row, weights, n_tokens, k, d, out_bf16, nullptr, (cudaStream_t)stream, false);
}

int b200q_moe_combine_chain(const b200q_moe_args* m, int n_tokens, float* add_to, cudaStream_t st) {
  return combine_launch(m->y, m->dest_row, m->weights, n_tokens, m->k, m->d, m->out, add_to, st, true);
}

// The two expert GEMMs on rows that are in their groups.
int b200q_moe_gemms_chain(const b200q_moe_args* m, int n_tokens, cudaStream_t st) {
  const int rows = b200q_moe_rows_max(n_tokens, m->n_experts, m->k);
  const int rc = b200q_mx_gemm_chain(m->a_q, m->a_e8, m->gu_q, m->gu_e8, m->off, m->ends, m->n_experts, rows, 2 * m->f, m->d, nullptr, m->act_q, m->act_e8, n_tokens, m->k, st);
  return rc != B200Q_OK ? rc : b200q_mx_gemm_chain(m->act_q, m->act_e8, m->dn_q, m->dn_e8, m->off, m->ends, m->n_experts, rows, m->d, m->f, m->y, nullptr, nullptr, n_tokens,
                                                   m->k, st);
}

// The expert layer in one call, its launches programmatic behind one another: route, dispatch + quantise, gate/up GEMM with SwiGLU + requantise, down GEMM,
// combine.  The GEMMs take the rows each expert has, not those its group is padded to.
int b200q_moe_layer_chain(const b200q_moe_args* m, const void* x_bf16, const float* logits, int n_tokens, float* add_to, cudaStream_t st, bool pdl) {
  if (!m || !x_bf16 || !logits || n_tokens <= 0 || !m->topi || !m->weights || !m->dest_row || !m->off || !m->ends || !m->scratch) return B200Q_ERR_BAD_ARG;
  if (m->n_experts <= 0 || m->k <= 0 || m->k > m->n_experts || (m->gating == 0 && m->mode != 0 && m->mode != 1)) return B200Q_ERR_BAD_ARG;
  if (m->gating && (m->gating < GATE_SOFTMAX || m->gating > GATE_SQRT_SOFTPLUS)) return B200Q_ERR_BAD_ARG;
  if (m->n_experts > 32 * MAX_E_PER_LANE || m->k > 32 || m->f % 128) return B200Q_ERR_BAD_SHAPE;
  int rc = route_launch(RouteRule{m->mode, m->gating, m->normalize, m->scale, m->sel_bias}, logits, n_tokens, m->n_experts, m->k, BLOCK_ROW, m->topi, m->weights, m->dest_row,
                        m->off, nullptr, m->ends, m->scratch, st, pdl);
  if (rc == B200Q_OK) rc = quantize_launch(x_bf16, B200Q_BF16, n_tokens, m->d, m->dest_row, m->k, m->a_q, m->a_e8, st, true);
  if (rc == B200Q_OK) rc = b200q_moe_gemms_chain(m, n_tokens, st);
  return rc == B200Q_OK ? combine_launch(m->y, m->dest_row, m->weights, n_tokens, m->k, m->d, m->out, add_to, st, true) : rc;
}
extern "C" int b200q_moe_layer(const b200q_moe_args* m, const void* x_bf16, const float* logits, int n_tokens, float* add_to, void* stream) {
  return b200q_moe_layer_chain(m, x_bf16, logits, n_tokens, add_to, (cudaStream_t)stream, false);
}
