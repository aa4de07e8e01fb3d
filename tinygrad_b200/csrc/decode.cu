// The non-GEMV kernels of one decode step: embedding lookup, one-token GQA attention
// with RoPE and KV-cache update, greedy arg-max.  Semantics follow
// tinygrad/llm/model.py:167-198 (attention, T == 1), :29-33 (RoPE), :358-364 (forward).
#include "common.cuh"
#include "actquant.cuh"
#include <math.h>

namespace {

// Sticky status of this file's kernels: 2 = a position outside [0, max_context) reached a kernel, which then skipped
// its work instead of reading or writing past the token table / KV cache.  b200q_status_read_clear reports it.
__device__ int g_decode_status = 0;

// Also leaves, for the first GEMV of the step, the row already multiplied by that GEMV's RMSNorm weight and
// quantised (actquant.cuh), with one partial sum of squares per block of 32.
__global__ void __launch_bounds__(256) embed_kernel(const __half* __restrict__ table, const int32_t* __restrict__ tokens,
                                                    const int32_t* __restrict__ pos, float* __restrict__ x, int dim, int vocab, int max_context,
                                                    void* xq_out, const __half* __restrict__ norm_w, float* ss_out) {
  pdl_launch_dependents();
  pdl_wait();
  int p = *pos;
  if (p < 0 || p > max_context) {      // the token table has max_context + 1 entries
    if (threadIdx.x == 0 && blockIdx.x == 0) atomicExch(&g_decode_status, 2);
    p = p < 0 ? 0 : max_context;       // keep the activations finite; the step's result is flagged invalid
  }
  int tok = tokens[p];
  tok = tok < 0 ? 0 : (tok >= vocab ? vocab - 1 : tok);
  const __half* row = table + (size_t)tok * dim;
  if (!xq_out) {
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < dim; i += gridDim.x * blockDim.x) x[i] = __half2float(row[i]);
    return;
  }
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, kgroups = (dim + GROUP_ELEMS - 1) / GROUP_ELEMS;
  const int wpb = blockDim.x >> 5;
  const XqDst dst(xq_out, kgroups);
  for (int b = blockIdx.x * wpb + warp; b < kgroups * 4; b += gridDim.x * wpb) {      // one warp per block of 32, lane = element
    const int k = b * 32 + lane;
    float v = 0.f;
    if (k < dim) { v = __half2float(row[k]); x[k] = v; }
    if (ss_out && b * 32 < dim) { const float s2 = warp_sum(v * v); if (lane == 0) ss_out[b] = s2; }
    quant_block_32x1((norm_w && k < dim) ? v * __half2float(norm_w[k]) : v, lane, b, dst);
  }
}

__global__ void advance_kernel(int32_t* pos, int max_context) {
  pdl_launch_dependents();
  pdl_wait();
  if (threadIdx.x == 0) {
    const int p = *pos;
    if (p < 0 || p >= max_context) atomicExch(&g_decode_status, 2);
    else *pos = p + 1;
  }
}

// ---------------------------------------------------------------------------
// attention.  grid (n_kv_heads, n_split); split s owns the fixed position range
// [s*ATTN_CHUNK, (s+1)*ATTN_CHUNK); CTAs past the current context leave at once.
// One warp per query head of the KV group.  The CTA first copies its K and V rows to
// shared memory with every thread's loads in flight together (one global latency), then
//   scores: each lane takes whole positions (full head_dim dot against the roped query),
//   values: each lane owns 4 consecutive head dims and walks the positions.
// Scratch layout:
//   float partial[n_heads][n_split][head_dim + 4]   (o[head_dim], running max, denominator, 2 pad)
//   uint  counter[n_kv_heads]                       (arrival count, reset by the last CTA)
constexpr int MAX_HD = 128;
constexpr int MAX_REP = 8;
#ifndef B200Q_ATTN_CHUNK
#define B200Q_ATTN_CHUNK 64
#endif
constexpr int ATTN_CHUNK = B200Q_ATTN_CHUNK;    // positions per CTA

template <typename KV> struct KvIO;
template <> struct KvIO<__half> {
  static constexpr int VEC = 8;   // elements per 16-byte word
  static __device__ __forceinline__ float dot(const __half* k, const float* q) {
    uint4 r = *reinterpret_cast<const uint4*>(k);
    float2 a = __half22float2(*reinterpret_cast<__half2*>(&r.x)), b = __half22float2(*reinterpret_cast<__half2*>(&r.y));
    float2 c = __half22float2(*reinterpret_cast<__half2*>(&r.z)), d = __half22float2(*reinterpret_cast<__half2*>(&r.w));
    return a.x * q[0] + a.y * q[1] + b.x * q[2] + b.y * q[3] + c.x * q[4] + c.y * q[5] + d.x * q[6] + d.y * q[7];
  }
  static __device__ __forceinline__ float4 load4(const __half* p) {
    uint2 r = *reinterpret_cast<const uint2*>(p);
    float2 a = __half22float2(*reinterpret_cast<__half2*>(&r.x)), b = __half22float2(*reinterpret_cast<__half2*>(&r.y));
    return make_float4(a.x, a.y, b.x, b.y);
  }
  static __device__ __forceinline__ __half cast(float v) { return __float2half_rn(v); }
};
template <> struct KvIO<float> {
  static constexpr int VEC = 4;
  static __device__ __forceinline__ float dot(const float* k, const float* q) {
    float4 r = *reinterpret_cast<const float4*>(k);
    return r.x * q[0] + r.y * q[1] + r.z * q[2] + r.w * q[3];
  }
  static __device__ __forceinline__ float4 load4(const float* p) { return *reinterpret_cast<const float4*>(p); }
  static __device__ __forceinline__ float cast(float v) { return v; }
};

__device__ __forceinline__ void cp_async16(void* smem_dst, const void* gmem_src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((uint32_t)__cvta_generic_to_shared(smem_dst)), "l"(gmem_src) : "memory");
}

#ifdef B200Q_GEMV_PROF
__device__ unsigned long long g_attn_prof[4096 * 8];
__device__ unsigned g_attn_prof_n;
__device__ __forceinline__ unsigned long long gtime() { unsigned long long t; asm volatile("mov.u64 %0, %globaltimer;" : "=l"(t)); return t; }
#define ASTAMP(i) do { if (threadIdx.x == 0) g_attn_prof[prof_slot * 8 + (i)] = gtime(); } while (0)
#else
#define ASTAMP(i) do {} while (0)
#endif

// Sequence blockIdx.z of a batch in lock-step: element strides between consecutive sequences (all zero for one sequence)
struct SeqStride { size_t qkv, cache, out, scratch_bytes; int pos; };

template <typename KV>
__global__ void __launch_bounds__(MAX_REP * 32) attn_decode_kernel(const b200q_attn_args a_in, const SeqStride sq) {
  constexpr int VEC = KvIO<KV>::VEC;
  b200q_attn_args a = a_in;
  if (blockIdx.z) {
    const size_t z = blockIdx.z;
    a.qkv += z * sq.qkv; a.out += z * sq.out; a.pos += z * sq.pos;
    a.k_cache = reinterpret_cast<KV*>(a.k_cache) + z * sq.cache; a.v_cache = reinterpret_cast<KV*>(a.v_cache) + z * sq.cache;
    a.scratch = reinterpret_cast<unsigned char*>(a.scratch) + z * sq.scratch_bytes;
  }
  extern __shared__ __align__(16) unsigned char asmem[];
  const int hd = a.head_dim, n_rep = a.n_heads / a.n_kv_heads, half_r = a.rope_dim >> 1;
  const int rstride = hd + VEC;                           // padded row: lanes reading different rows hit different banks
  KV* s_k = reinterpret_cast<KV*>(asmem);                 // [ATTN_CHUNK][rstride]
  KV* s_v = s_k + ATTN_CHUNK * rstride;                   // [ATTN_CHUNK][rstride]
  float* s_q = reinterpret_cast<float*>(s_v + ATTN_CHUNK * rstride);   // [n_rep][hd] roped queries
  float* s_sc = s_q + n_rep * hd;                         // [n_rep][ATTN_CHUNK] scores, then probabilities
  float* s_part = s_sc + n_rep * ATTN_CHUNK;              // [n_rep][hd + 4] what a head's second warp hands to its first (rows stay 16-byte aligned)
  __shared__ int s_last;
  const int kvh = blockIdx.x, split = blockIdx.y;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#ifdef B200Q_GEMV_PROF
  __shared__ unsigned s_prof_slot;
  if (threadIdx.x == 0) {
    s_prof_slot = (unsigned)a.flags >> 16;           // experiment builds: the host puts the launch's slot into the upper half of flags
    if (blockIdx.x == 0 && blockIdx.y == 0) g_attn_prof[s_prof_slot * 8 + 0] = gtime();
  }
  __syncthreads();
  const unsigned prof_slot = s_prof_slot;
  const bool prof_cta = blockIdx.x == 0 && blockIdx.y == 0;
#endif
  pdl_launch_dependents();
  const int lo = split * ATTN_CHUNK;
  KV* kc = reinterpret_cast<KV*>(a.k_cache) + (size_t)kvh * a.max_context * hd;
  KV* vc = reinterpret_cast<KV*>(a.v_cache) + (size_t)kvh * a.max_context * hd;
  // All cached rows of the slice -> shared memory with asynchronous 16-byte copies: every copy of the CTA is in flight at once
  // (one global latency).  The rows were written by earlier steps, so the copies are issued BEFORE the wait for the previous
  // kernel (they overlap its tail); only the position counter they are sized by could, in principle, still be the previous
  // step's, so it is read again after the wait and the copies are redone in the (never observed) case that it moved.
  auto fetch_rows = [&](int pos_now) {
    const int wpr = hd / VEC, n_old = max(0, min(min(ATTN_CHUNK, a.max_context - lo), pos_now - lo)), words = n_old * wpr;
    for (int i = threadIdx.x; i < words; i += blockDim.x) {
      const int r = i / wpr, c = (i - r * wpr) * VEC;
      cp_async16(s_k + r * rstride + c, kc + (size_t)(lo + r) * hd + c);
      cp_async16(s_v + r * rstride + c, vc + (size_t)(lo + r) * hd + c);
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  const int pos_early = min(max(__ldcg(a.pos), 0), a.max_context - 1);
  if (threadIdx.x * 32 < a.rope_dim) prefetch_l2(a.rope + (size_t)pos_early * a.rope_dim + threadIdx.x * 32);
  fetch_rows(pos_early);
  pdl_wait();
#ifdef B200Q_GEMV_PROF
  if (prof_cta) ASTAMP(1);
#endif
  const int pos = __ldcg(a.pos);
  if (pos < 0 || pos >= a.max_context) {        // no cache row for this position: touch nothing (uniform over the grid)
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    if (threadIdx.x == 0) atomicExch(&g_decode_status, 2);
    return;
  }
  if (pos != pos_early) {                       // uniform over the CTA
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    __syncthreads();
    fetch_rows(pos);
  }
#ifdef B200Q_GEMV_PROF
  if (prof_cta) ASTAMP(5);
#endif
  const int n_ctx = pos + 1;
  if (lo >= n_ctx) { asm volatile("cp.async.wait_group 0;" ::: "memory"); return; }
  const int n = min(ATTN_CHUNK, n_ctx - lo);
  const int n_active = (n_ctx + ATTN_CHUNK - 1) / ATTN_CHUNK;
  // RoPE, half-split layout: (x1 cos - x2 sin) || (x2 cos + x1 sin); dims past rope_dim pass through
  const float* rope = a.rope + (size_t)pos * a.rope_dim;
  for (int i = threadIdx.x; i < n_rep * hd; i += blockDim.x) {
    const int r = i / hd, d = i - r * hd;
    const float* q = a.qkv + (size_t)(kvh * n_rep + r) * hd;
    float v = q[d];
    if (d < half_r) v = q[d] * rope[d] - q[d + half_r] * rope[half_r + d];
    else if (d < a.rope_dim) v = q[d] * rope[d - half_r] + q[d - half_r] * rope[d];
    s_q[i] = v;
  }
  if (lo <= pos && pos < lo + ATTN_CHUNK) {   // this CTA owns the new position: append it to the cache and to its slice
    const float* kq = a.qkv + (size_t)a.n_heads * hd + (size_t)kvh * hd;
    const float* vq = a.qkv + (size_t)(a.n_heads + a.n_kv_heads) * hd + (size_t)kvh * hd;
    for (int d = threadIdx.x; d < hd; d += blockDim.x) {
      float v = kq[d];
      if (d < half_r) v = kq[d] * rope[d] - kq[d + half_r] * rope[half_r + d];
      else if (d < a.rope_dim) v = kq[d] * rope[d - half_r] + kq[d - half_r] * rope[d];
      const KV kk = KvIO<KV>::cast(v), vv = KvIO<KV>::cast(vq[d]);
      kc[(size_t)pos * hd + d] = kk; vc[(size_t)pos * hd + d] = vv;
      s_k[(pos - lo) * rstride + d] = kk; s_v[(pos - lo) * rstride + d] = vv;
    }
  }
  asm volatile("cp.async.wait_group 0;" ::: "memory");
  __syncthreads();
#ifdef B200Q_GEMV_PROF
  if (prof_cta) ASTAMP(6);
#endif

  const int d0 = lane * 4;
  const bool dl = d0 < hd;
  const float scale = 1.0f / sqrtf((float)hd);
  float* partial = reinterpret_cast<float*>(a.scratch);
  const int pstride = hd + 4;   // keeps every record 16-byte aligned
  // A head's positions are shared by `ws` warps (blockDim = ws * n_rep warps; ws = 2 when the block has room): warp w works on head
  // w % n_rep and on the positions 32 * (w / n_rep) + 32 * ws * j + lane.  Each has its own running max / denominator / output; the
  // head's first warp merges them (the same merge as across slices) and carries on alone.
  const int ws = (int)(blockDim.x >> 5) / n_rep, head = warp % n_rep, part = warp / n_rep;
  float mx = -INFINITY, den = 0.f;
  float4 o = make_float4(0, 0, 0, 0);
  {
    float* sc = s_sc + head * ATTN_CHUNK;
    const float* q = s_q + head * hd;
    float lmax = -INFINITY;
    for (int i = 32 * part + lane; i < n; i += 32 * ws) {
      const KV* kr = s_k + i * rstride;
      // four running sums: a lane's dot product is a dependent chain otherwise
      float s0 = 0.f, s1 = 0.f, s2 = 0.f, s3 = 0.f;
      int d = 0;
      for (; d + 4 * VEC <= hd; d += 4 * VEC) {
        s0 += KvIO<KV>::dot(kr + d, q + d); s1 += KvIO<KV>::dot(kr + d + VEC, q + d + VEC);
        s2 += KvIO<KV>::dot(kr + d + 2 * VEC, q + d + 2 * VEC); s3 += KvIO<KV>::dot(kr + d + 3 * VEC, q + d + 3 * VEC);
      }
      for (; d < hd; d += VEC) s0 += KvIO<KV>::dot(kr + d, q + d);
      float s = (s0 + s1) + (s2 + s3);
      s *= scale;
      sc[i] = s;
      lmax = fmaxf(lmax, s);
    }
    mx = warp_max(lmax);
    float lsum = 0.f;
    for (int i = 32 * part + lane; i < n; i += 32 * ws) { const float pr = __expf(sc[i] - mx); sc[i] = pr; lsum += pr; }
    den = warp_sum(lsum);
    __syncwarp();
    if (dl) {
      const KV* vr = s_v + d0;
      float4 o2 = make_float4(0, 0, 0, 0);      // two independent sums
      for (int b0 = 32 * part; b0 < n; b0 += 32 * ws) {      // this warp's runs of 32 positions
        const int e = min(n, b0 + 32);
        int i = b0;
#pragma unroll 4
        for (; i + 2 <= e; i += 2) {
          const float pr = sc[i], pr2 = sc[i + 1];
          const float4 v = KvIO<KV>::load4(vr + i * rstride), v2 = KvIO<KV>::load4(vr + (i + 1) * rstride);
          o.x = fmaf(pr, v.x, o.x); o.y = fmaf(pr, v.y, o.y); o.z = fmaf(pr, v.z, o.z); o.w = fmaf(pr, v.w, o.w);
          o2.x = fmaf(pr2, v2.x, o2.x); o2.y = fmaf(pr2, v2.y, o2.y); o2.z = fmaf(pr2, v2.z, o2.z); o2.w = fmaf(pr2, v2.w, o2.w);
        }
        if (i < e) {
          const float pr = sc[i];
          const float4 v = KvIO<KV>::load4(vr + i * rstride);
          o.x = fmaf(pr, v.x, o.x); o.y = fmaf(pr, v.y, o.y); o.z = fmaf(pr, v.z, o.z); o.w = fmaf(pr, v.w, o.w);
        }
      }
      o.x += o2.x; o.y += o2.y; o.z += o2.z; o.w += o2.w;
    }
  }
  if (ws > 1) {
    float* hp = s_part + head * (hd + 4);
    if (part == 1) {
      if (dl) *reinterpret_cast<float4*>(hp + d0) = o;
      if (lane == 0) { hp[hd] = mx; hp[hd + 1] = den; }
    }
    __syncthreads();
    if (part == 0) {
      const float m1 = hp[hd], l1 = hp[hd + 1];
      const float gm = fmaxf(mx, m1);                       // the first warp always holds position 0 of the slice: mx is finite
      const float c0 = __expf(mx - gm), c1 = l1 > 0.f ? __expf(m1 - gm) : 0.f;
      float4 o1 = make_float4(0, 0, 0, 0);
      if (dl) o1 = *reinterpret_cast<const float4*>(hp + d0);
      o.x = o.x * c0 + o1.x * c1; o.y = o.y * c0 + o1.y * c1; o.z = o.z * c0 + o1.z * c1; o.w = o.w * c0 + o1.w * c1;
      den = den * c0 + l1 * c1;
      mx = gm;
    }
  }
  if (part == 0) {
    if (n_active == 1) {   // short context: this CTA holds the whole softmax
      const float inv = 1.f / den;
      const float4 r = make_float4(o.x * inv, o.y * inv, o.z * inv, o.w * inv);
      if (dl) *reinterpret_cast<float4*>(a.out + (size_t)(kvh * n_rep + head) * hd + d0) = r;
      if (a.xq_out) quant_block_8x4(r, lane & 7, (kvh * n_rep + head) * 4 + (lane >> 3), XqDst(a.xq_out, a.n_heads));   // head_dim 128: one group per head
    } else {
      float* pp = partial + ((size_t)(kvh * n_rep + head) * a.n_split + split) * pstride;
      if (dl) *reinterpret_cast<float4*>(pp + d0) = o;
      if (lane == 0) { pp[hd] = mx; pp[hd + 1] = den; }
    }
  }
  if (n_active == 1) return;
#ifdef B200Q_GEMV_PROF
  if (prof_cta) ASTAMP(2);
  if (threadIdx.x == 0) atomicMax(&g_attn_prof[prof_slot * 8 + 7], gtime());      // this slot is re-used: max over CTAs of "partials done"
#endif
  // last CTA of this KV head merges the slices
  __threadfence();
  __syncthreads();
  unsigned* counter = reinterpret_cast<unsigned*>(partial + (size_t)a.n_heads * a.n_split * pstride);
  if (threadIdx.x == 0) {
    const unsigned prev = atomicAdd(&counter[kvh], 1u);
    s_last = (prev == (unsigned)n_active - 1);
    if (s_last) counter[kvh] = 0;
  }
  __syncthreads();
  if (!s_last) return;
  __threadfence();
#ifdef B200Q_GEMV_PROF
  if (kvh == 0) { if (threadIdx.x == 0) g_attn_prof[prof_slot * 8 + 3] = gtime(); }
#endif
  if (warp < n_rep) {
    const float* hp = partial + (size_t)(kvh * n_rep + warp) * a.n_split * pstride;
    // Batches of 16 slices: the statistics (one slice per lane) and every lane's 4 output dims of all 16 slices are
    // loaded before anything is used, so a batch costs one L2 round trip.  Running max / denominator across batches.
    float gm = -INFINITY, den = 0.f;
    float4 o = make_float4(0, 0, 0, 0);
    for (int s0 = 0; s0 < n_active; s0 += 16) {
      const int cnt = min(16, n_active - s0);
      float2 ml = make_float2(-INFINITY, 0.f);
      if (lane < cnt) ml = __ldcg(reinterpret_cast<const float2*>(hp + (size_t)(s0 + lane) * pstride + hd));
      float4 ov[16];
#pragma unroll
      for (int j = 0; j < 16; j++)
        ov[j] = (dl && j < cnt) ? __ldcg(reinterpret_cast<const float4*>(hp + (size_t)(s0 + j) * pstride + d0)) : make_float4(0, 0, 0, 0);
      const float nm = fmaxf(gm, warp_max(ml.x));
      const float corr = __expf(gm - nm);
      const float w = lane < cnt ? __expf(ml.x - nm) : 0.f;
      den = den * corr + warp_sum(w * ml.y);
      o.x *= corr; o.y *= corr; o.z *= corr; o.w *= corr;
#pragma unroll
      for (int j = 0; j < 16; j++) {
        const float wj = __shfl_sync(0xffffffffu, w, j);      // every lane takes part in the shuffle
        o.x = fmaf(wj, ov[j].x, o.x); o.y = fmaf(wj, ov[j].y, o.y); o.z = fmaf(wj, ov[j].z, o.z); o.w = fmaf(wj, ov[j].w, o.w);
      }
      gm = nm;
    }
    const float inv = 1.f / den;
    const float4 r = make_float4(o.x * inv, o.y * inv, o.z * inv, o.w * inv);
    if (dl) *reinterpret_cast<float4*>(a.out + (size_t)(kvh * n_rep + warp) * hd + d0) = r;
    if (a.xq_out) quant_block_8x4(r, lane & 7, (kvh * n_rep + warp) * 4 + (lane >> 3), XqDst(a.xq_out, a.n_heads));
  }
#ifdef B200Q_GEMV_PROF
  if (kvh == 0) { __syncthreads(); if (threadIdx.x == 0) g_attn_prof[prof_slot * 8 + 4] = gtime(); }
#endif
}

#ifdef B200Q_GEMV_PROF
}  // namespace
extern "C" int b200q_attn_prof_read(unsigned long long* out, int max_slots, unsigned* n) {
  B200Q_CHECK_CUDA(cudaMemcpyFromSymbol(out, g_attn_prof, sizeof(unsigned long long) * 8 * (max_slots < 4096 ? max_slots : 4096)));
  B200Q_CHECK_CUDA(cudaMemcpyFromSymbol(n, g_attn_prof_n, sizeof(unsigned)));
  return B200Q_OK;
}
extern "C" int b200q_attn_prof_reset(void) {
  static unsigned long long zeros[4096 * 8];
  B200Q_CHECK_CUDA(cudaMemcpyToSymbol(g_attn_prof, zeros, sizeof(zeros)));
  return B200Q_OK;
}
namespace {
#endif

// ---------------------------------------------------------------------------
// The same attention for head_dim 64 / 128: one thread-block cluster of 8 or 16 CTAs per KV head.
//
// What bounds it: at a few hundred positions nothing but latency.  In the kernel above (8B shape, position 520: 8.4 us from the row's arrival
// to the last store; 10.4 us of a block with its launch, 6.5 now) 3.4 us went into dot products of one lane per position and head, which read every cached row once per query head, and
// 3 us into merging slices through global memory (fence, counter, two dependent rounds of loads).  Here
//  * the query heads of the KV head are the rows of a tensor-core operand, their fp16 high parts in rows 0..7 and the remainders in rows
//    8..15: one m16n8k16 product gives both, a cached row is read once for all heads; the probabilities go into the second product the
//    same way, so that only the cache dtype rounds (as in the prompt kernel);
//  * the positions are split over the cluster's CTAs in whole chunks of 64; the CTAs' partial results meet in distributed shared memory: one
//    cluster barrier and one round of remote loads.  The split follows the position, so contexts of any length are spread over all CTAs;
//  * two chunks at a time: keys and values of the first two are on their way before the wait for the previous kernel, the next two's keys go out when this round's scores are
//    there, its values when they are used.  One chunk a round, two in flight: 12.3 us at 3507 positions of 28 / 4 heads (4 chunks a CTA; a launch, in order), 10.3; 14.3, 12.3 with 32 / 8;
//  * after the wait one round trip through L2: the position comes with the values of q, k and v, cosines and sines are there already (position, then all of these: 8B
//    Q4_0 10390 us for 8 tokens at 512, 10118); the last cluster barrier is entered at the last remote load, not after the output's store.
// fp32 caches: the same with m16n8k8 tf32 products.  Queries, probabilities and cached values are all split in two tf32 numbers (2^-22 of the value
// together, with the range of fp32), a cached value on its way from shared memory to the operand.
constexpr int AC_THREADS = 256, AC_POS = 64, AC_ROUND = 2 * AC_POS;
template <int HD, typename KV> struct AcSmem {           // bytes; rows padded so that fragment loads hit distinct banks
  static constexpr bool F32 = sizeof(KV) == 4;
  static constexpr int KROW = F32 ? (HD + 4) * 4 : (HD + 8) * 2, VROW = (HD + 8) * (int)sizeof(KV), QROW = KROW, PROW = F32 ? (AC_ROUND + 4) * 4 : (AC_ROUND + 8) * 2;
  static constexpr int V = AC_ROUND * KROW, Q = V + AC_ROUND * VROW, P = Q + 16 * QROW, S = P + 16 * PROW, O = S + 8 * (AC_ROUND + 4) * 4, ST = O + 8 * HD * 4, TOTAL = ST + 8 * 4 * 4;
};

__device__ __forceinline__ void mma_f16(float (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
               : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3]) : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
__device__ __forceinline__ void mma_tf32(float (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  asm volatile("mma.sync.aligned.m16n8k8.row.col.f32.tf32.tf32.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
               : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3]) : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
// The same for operands whose rows 8 .. 15 hold what the rounding of rows 0 .. 7 left: the sums of rows 0 .. 7 are added here, to nearest.  The tensor core
// truncates, always towards zero, when it adds to an accumulator.  Error of the output's norm against 64 bits, 37 .. 3507 positions (root mean square of 64
// cases): fp16 caches 2.0e-7 (2.2e-7 with probabilities of at most 1), with running accumulators 3.1e-7; fp32 caches 2.2e-7, 8.6e-7 (up to 2.4e-6); the one-lane-per-position kernel 2.0e-7.
__device__ __forceinline__ void mma_f16_rn(float (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  float p[4] = {0.f, 0.f, c[2], c[3]};
  mma_f16(p, a, b0, b1);
  c[0] += p[0]; c[1] += p[1]; c[2] = p[2]; c[3] = p[3];
}
// ... with the second operand as a sum, h + l
__device__ __forceinline__ void mma_tf32_rn(float (&c)[4], const uint32_t (&a)[4], uint32_t h0, uint32_t h1, uint32_t l0, uint32_t l1) {
  float p[4] = {0.f, 0.f, c[2], c[3]};
  mma_tf32(p, a, l0, l1);
  mma_tf32(p, a, h0, h1);
  c[0] += p[0]; c[1] += p[1]; c[2] = p[2]; c[3] = p[3];
}
// tf32 high part and the remainder's tf32 rounding (both are valid fp32 bit patterns)
__device__ __forceinline__ void split_tf32(float v, uint32_t& hi, uint32_t& lo) {
  asm("cvt.rna.tf32.f32 %0, %1;" : "=r"(hi) : "f"(v));
  asm("cvt.rna.tf32.f32 %0, %1;" : "=r"(lo) : "f"(v - __uint_as_float(hi)));
}
__device__ __forceinline__ void ldsm4(uint32_t (&r)[4], uint32_t addr) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr) : "memory");
}
__device__ __forceinline__ void ldsm4t(uint32_t (&r)[4], uint32_t addr) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr) : "memory");
}
// fp16 high part and the remainder's fp16 rounding
__device__ __forceinline__ void split_h(float v, __half& hi, __half& lo) {
  hi = __float2half_rn(v);
  lo = __float2half_rn(v - __half2float(hi));
}

// value d of a row, split in two rows of operand values
template <typename KV> __device__ __forceinline__ void store_split(float v, unsigned char* hi_row, unsigned char* lo_row, int d) {
  if constexpr (sizeof(KV) == 4) {
    split_tf32(v, reinterpret_cast<uint32_t*>(hi_row)[d], reinterpret_cast<uint32_t*>(lo_row)[d]);
  } else {
    __half hi, lo;
    split_h(v, hi, lo);
    reinterpret_cast<__half*>(hi_row)[d] = hi; reinterpret_cast<__half*>(lo_row)[d] = lo;
  }
}
// a load that is issued where it stands
__device__ __forceinline__ float ld_now(const float* p) {
  float v;
  asm volatile("ld.global.cg.f32 %0, [%1];" : "=f"(v) : "l"(p) : "memory");
  return v;
}
template <typename KV> __device__ __forceinline__ KV cache_cast(float v);
template <> __device__ __forceinline__ __half cache_cast<__half>(float v) { return __float2half_rn(v); }
template <> __device__ __forceinline__ float cache_cast<float>(float v) { return v; }
// m16n8k8 A fragment: rows g and g + 8 (`down` bytes on), columns t and t + 4
__device__ __forceinline__ void ld_frag_tf32(uint32_t (&r)[4], const unsigned char* at, int down) {
  r[0] = *reinterpret_cast<const uint32_t*>(at); r[1] = *reinterpret_cast<const uint32_t*>(at + down);
  r[2] = *reinterpret_cast<const uint32_t*>(at + 16); r[3] = *reinterpret_cast<const uint32_t*>(at + down + 16);
}

template <int HD, int CL, typename KV>      // CL: CTAs per cluster
__global__ void __launch_bounds__(AC_THREADS) attn_cluster_kernel(const b200q_attn_args a_in, const SeqStride sq) {
  using M = AcSmem<HD, KV>;
  constexpr bool F32 = M::F32;
  constexpr int VEC = 16 / sizeof(KV), ROW_VECS = HD / VEC;         // cache elements per 16 bytes, 16-byte pieces per row
  extern __shared__ __align__(16) unsigned char asmem[];
  b200q_attn_args a = a_in;
  if (blockIdx.z) {
    const size_t z = blockIdx.z;
    a.qkv += z * sq.qkv; a.out += z * sq.out; a.pos += z * sq.pos;
    a.k_cache = reinterpret_cast<KV*>(a.k_cache) + z * sq.cache; a.v_cache = reinterpret_cast<KV*>(a.v_cache) + z * sq.cache;
  }
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, g = lane >> 2, t = lane & 3;
  const int kvh = blockIdx.x, rank = blockIdx.y, n_rep = a.n_heads / a.n_kv_heads, half_r = a.rope_dim >> 1;
  const uint32_t base = (uint32_t)__cvta_generic_to_shared(asmem);
  float* s_s = reinterpret_cast<float*>(asmem + M::S);            // [8][128 + 4] scores
  float* s_o = reinterpret_cast<float*>(asmem + M::O);            // [8][HD] this CTA's unnormalised output
  float* s_m = reinterpret_cast<float*>(asmem + M::ST);           // [8] running max, [8] denominator, [8] rescale factor
  float *s_l = s_m + 8, *s_c = s_m + 16, *s_q = s_m + 24;        // [8] what a head's scores are multiplied with
  KV* kc = reinterpret_cast<KV*>(a.k_cache) + (size_t)kvh * a.max_context * HD;
  KV* vc = reinterpret_cast<KV*>(a.v_cache) + (size_t)kvh * a.max_context * HD;
  pdl_launch_dependents();
  int c0 = 0, c1 = 0;
  // cached rows of the round that starts with chunk `ch`, of K or of V (asynchronously, one commit group; chunks past c1: an empty one)
  auto fetch = [&](int ch, const KV* from, int to, int row, int pos_now) {
    const int n_old = min(AC_ROUND, min(c1 * AC_POS, pos_now) - ch * AC_POS);
    for (int i = tid; i < n_old * ROW_VECS; i += AC_THREADS) {
      const int r = i / ROW_VECS, c = i - r * ROW_VECS;
      cp_async16(asmem + to + r * row + c * 16, from + (size_t)(ch * AC_POS + r) * HD + c * VEC);
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  auto start = [&](int pos_now) {                                  // this CTA's chunks for a context of pos_now + 1 positions, and the first round's copies
    const int n_chunks = pos_now / AC_POS + 1, per = (n_chunks + CL - 1) / CL;
    c0 = min(n_chunks, rank * per); c1 = min(n_chunks, c0 + per);
    fetch(c0, kc, 0, M::KROW, pos_now);
    fetch(c0, vc, M::V, M::VROW, pos_now);
  };
  // The rows were written by earlier steps: the copies go out before the wait for the previous kernel.  The position they are sized by is read
  // again after it, and the copies are redone in the (never observed) case that it moved.
  const int pos_early = min(max(__ldcg(a.pos), 0), a.max_context - 1);
  start(pos_early);
  for (int i = tid; i < (16 * M::QROW + 16 * M::PROW) / 16; i += AC_THREADS) reinterpret_cast<uint4*>(asmem + M::Q)[i] = make_uint4(0, 0, 0, 0);   // rows of absent heads
  if (tid < 8) { s_m[tid] = -INFINITY; s_l[tid] = 0.f; s_q[tid] = 0.f; }
  // RoPE, half-split layout: (x1 cos - x2 sin) || (x2 cos + x1 sin); dims past rope_dim pass through.  The table does not change: cosine and sine of the dims of this thread's
  // query values and of its value of the new K row are read before the wait, too.
  constexpr int QV = HD / 32;
  float2 q_rot[QV], k_rot;
  auto rotation = [&](int d, int pos_now) {
    const float* rope = a.rope + (size_t)pos_now * a.rope_dim;
    return d < half_r ? make_float2(rope[d], rope[d + half_r]) : d < a.rope_dim ? make_float2(rope[d - half_r], rope[d]) : make_float2(1.f, 0.f);
  };
  auto rotations = [&](int pos_now) {
#pragma unroll
    for (int j = 0; j < QV; j++) q_rot[j] = rotation(lane + 32 * j, pos_now);
    k_rot = rotation(tid % HD, pos_now);
  };
  auto partner = [&](int d) { return d < half_r ? d + half_r : d < a.rope_dim ? d - half_r : d; };
  auto roped = [&](float v, float other, float2 r, int d) {
    if (d < half_r) return v * r.x - other * r.y;
    if (d < a.rope_dim) return v * r.x + other * r.y;
    return v;
  };
  rotations(pos_early);
  __syncthreads();
  pdl_wait();
  // one round trip: the position, and the values that do not hang on it (a warp takes a query head; a thread a value of the new K row and one of the new V row)
  int pos;
  asm volatile("ld.global.cg.s32 %0, [%1];" : "=r"(pos) : "l"(a.pos) : "memory");
  const float *q_row = a.qkv + (size_t)(kvh * n_rep + warp) * HD, *k_row = a.qkv + (size_t)(a.n_heads + kvh) * HD, *v_row = k_row + (size_t)a.n_kv_heads * HD;
  float q[QV], q_other[QV], k_new = 0.f, k_other = 0.f, v_new = 0.f;
  if (warp < n_rep)
#pragma unroll
    for (int j = 0; j < QV; j++) { q[j] = ld_now(q_row + lane + 32 * j); q_other[j] = ld_now(q_row + partner(lane + 32 * j)); }
  if (tid < HD) { k_new = ld_now(k_row + tid); k_other = ld_now(k_row + partner(tid)); v_new = ld_now(v_row + tid); }
  if (pos < 0 || pos >= a.max_context) {                           // no cache row for this position: touch nothing (uniform over the cluster)
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    if (tid == 0 && rank == 0) atomicExch(&g_decode_status, 2);
    return;
  }
  if (pos != pos_early) {
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    __syncthreads();
    start(pos);
    rotations(pos);
  }
  const bool owner = c0 < c1 && pos / AC_POS == c1 - 1;             // the new position is in this CTA's last chunk
  if (c0 < c1 && warp < n_rep) {                                   // fp16: under a power of two of the head's own
    float up = 1.f, down = 1.f;
#pragma unroll
    for (int j = 0; j < QV; j++) q[j] = roped(q[j], q_other[j], q_rot[j], lane + 32 * j);
    if constexpr (!F32) {
      float amax = 0.f;
#pragma unroll
      for (int j = 0; j < QV; j++) amax = fmaxf(amax, fabsf(q[j]));
      pow2_scale(warp_max(amax), up, down);
    }
#pragma unroll
    for (int j = 0; j < QV; j++) store_split<KV>(q[j] * up, asmem + M::Q + warp * M::QROW, asmem + M::Q + (8 + warp) * M::QROW, lane + 32 * j);
    if (lane == 0) s_q[warp] = down * (1.0f / sqrtf((float)HD));
  }
  const KV k_cast = cache_cast<KV>(roped(k_new, k_other, k_rot, tid)), v_cast = cache_cast<KV>(v_new);
  if (owner && tid < HD) { kc[(size_t)pos * HD + tid] = k_cast; vc[(size_t)pos * HD + tid] = v_cast; }
  float acc[HD / 64][4];                                             // this warp's HD / 8 output dims: rows g (high parts) and g + 8 (low parts)
#pragma unroll
  for (int j = 0; j < HD / 64; j++) acc[j][0] = acc[j][1] = acc[j][2] = acc[j][3] = 0.f;
  for (int ch = c0; ch < c1; ch += 2) {
    const bool two = ch + 1 < c1;
    const int end = two ? AC_ROUND : AC_POS, nv = min(end, pos + 1 - ch * AC_POS);
    if (nv < end || (owner && ch + 2 >= c1)) {                       // the last chunk: append the new row, and no stale values behind it (0 * NaN)
      if (tid < HD) {
        *reinterpret_cast<KV*>(asmem + (nv - 1) * M::KROW + tid * (int)sizeof(KV)) = k_cast;
        *reinterpret_cast<KV*>(asmem + M::V + (nv - 1) * M::VROW + tid * (int)sizeof(KV)) = v_cast;
      }
      for (int i = tid; i < (end - nv) * ROW_VECS; i += AC_THREADS)
        *reinterpret_cast<uint4*>(asmem + M::V + (nv + i / ROW_VECS) * M::VROW + (i % ROW_VECS) * 16) = make_uint4(0, 0, 0, 0);
    }
    asm volatile("cp.async.wait_group 1;" ::: "memory");             // the keys
    __syncthreads();                                                 // (also: queries and the new rows are in place)
#pragma unroll 1
    for (int p0 = 0; p0 < end; p0 += AC_POS) {                       // scores: warp w takes positions 8w .. 8w + 7 of a chunk
      float c[4] = {0.f, 0.f, 0.f, 0.f}, c2[4] = {0.f, 0.f, 0.f, 0.f};
      const unsigned char* kr = asmem + (p0 + warp * 8 + g) * M::KROW + t * 4;
      if constexpr (F32) {
        const unsigned char* qa = asmem + M::Q + g * M::QROW + t * 4;
#pragma unroll 4
        for (int kk = 0; kk < HD / 8; kk++) {
          uint32_t q4[4], h0, l0, h1, l1;
          ld_frag_tf32(q4, qa + kk * 32, 8 * M::QROW);
          split_tf32(*reinterpret_cast<const float*>(kr + kk * 32), h0, l0);
          split_tf32(*reinterpret_cast<const float*>(kr + kk * 32 + 16), h1, l1);
          if (kk & 1) mma_tf32_rn(c2, q4, h0, h1, l0, l1); else mma_tf32_rn(c, q4, h0, h1, l0, l1);
        }
      } else {
        const uint32_t qa = base + M::Q + (lane & 15) * M::QROW + (lane >> 4) * 16;
#pragma unroll
        for (int kk = 0; kk < HD / 16; kk++) {
          uint32_t q4[4];
          ldsm4(q4, qa + kk * 32);
          const uint32_t b0 = *reinterpret_cast<const uint32_t*>(kr + kk * 32), b1 = *reinterpret_cast<const uint32_t*>(kr + kk * 32 + 16);
          if (kk & 1) mma_f16_rn(c2, q4, b0, b1); else mma_f16_rn(c, q4, b0, b1);
        }
      }
      const int p = p0 + warp * 8 + 2 * t;
      const float scale = s_q[g], s0 = ((c[0] + c2[0]) + (c[2] + c2[2])) * scale, s1 = ((c[1] + c2[1]) + (c[3] + c2[3])) * scale;
      s_s[g * (AC_ROUND + 4) + p] = p < nv ? s0 : -INFINITY;
      s_s[g * (AC_ROUND + 4) + p + 1] = p + 1 < nv ? s1 : -INFINITY;
    }
    __syncthreads();
    fetch(ch + 2, kc, 0, M::KROW, pos);                              // the next round's keys, while this one's probabilities are made and used
    if (warp < n_rep) {                                              // softmax of head `warp`
      constexpr float UP = F32 ? 1.f : 256.f;                        // probabilities (and their sum) 256 times as large: a remainder below 2^-14 loses bits
      const float* sc = s_s + warp * (AC_ROUND + 4) + 2 * lane;
      const float2 s2 = *reinterpret_cast<const float2*>(sc), s3 = two ? *reinterpret_cast<const float2*>(sc + AC_POS) : make_float2(-INFINITY, -INFINITY);
      const float m0 = s_m[warp], m1 = fmaxf(m0, warp_max(fmaxf(fmaxf(s2.x, s2.y), fmaxf(s3.x, s3.y))));
      const float cr = __expf(m0 - m1), p[4] = {__expf(s2.x - m1) * UP, __expf(s2.y - m1) * UP, __expf(s3.x - m1) * UP, __expf(s3.y - m1) * UP}, sum = warp_sum((p[0] + p[1]) + (p[2] + p[3]));
#pragma unroll
      for (int j = 0; j < 4; j += 2) {
        unsigned char* const pr = asmem + M::P + warp * M::PROW;
        const int at = 2 * lane + j / 2 * AC_POS;
        if constexpr (F32) {
          store_split<KV>(p[j], pr, pr + 8 * M::PROW, at);
          store_split<KV>(p[j + 1], pr, pr + 8 * M::PROW, at + 1);
        } else {
          __half h0, l0, h1, l1;
          split_h(p[j], h0, l0); split_h(p[j + 1], h1, l1);
          *reinterpret_cast<__half2*>(pr + at * 2) = __halves2half2(h0, h1);
          *reinterpret_cast<__half2*>(pr + 8 * M::PROW + at * 2) = __halves2half2(l0, l1);
        }
      }
      __syncwarp();
      if (lane == 0) { s_m[warp] = m1; s_l[warp] = s_l[warp] * cr + sum; s_c[warp] = cr; }
    }
    asm volatile("cp.async.wait_group 1;" ::: "memory");             // the values
    __syncthreads();
    const float cr = g < n_rep ? s_c[g] : 0.f;
#pragma unroll
    for (int j = 0; j < HD / 64; j++) { acc[j][0] *= cr; acc[j][1] *= cr; acc[j][2] *= cr; acc[j][3] *= cr; }
#pragma unroll 1
    for (int p0 = 0; p0 < end; p0 += AC_POS) {                       // O = P V: warp w takes HD / 8 dims
      if constexpr (F32) {
        const unsigned char *pa = asmem + M::P + g * M::PROW + (p0 + t) * 4, *va = asmem + M::V + (p0 + t) * M::VROW + (warp * (HD / 8) + g) * 4;
#pragma unroll 4
        for (int kk = 0; kk < AC_POS / 8; kk++) {
          uint32_t p4[4];
          ld_frag_tf32(p4, pa + kk * 32, 8 * M::PROW);
#pragma unroll
          for (int j = 0; j < HD / 64; j++) {
            uint32_t h0, l0, h1, l1;
            split_tf32(*reinterpret_cast<const float*>(va + kk * 8 * M::VROW + j * 32), h0, l0);
            split_tf32(*reinterpret_cast<const float*>(va + (kk * 8 + 4) * M::VROW + j * 32), h1, l1);
            mma_tf32_rn(acc[j], p4, h0, h1, l0, l1);
          }
        }
      } else {
      const uint32_t pa = base + M::P + (lane & 15) * M::PROW + (lane >> 4) * 16 + p0 * 2;
      // transposing loads: 8x8 blocks of (positions, dims).  128: positions kk*16 + {0..7, 8..15} x dims {0..7, 8..15}; 64: 32 positions x 8 dims
      const uint32_t va = base + M::V + p0 * M::VROW + warp * (HD / 8) * 2 +
                          (HD == 128 ? (((lane >> 3) & 1) * 8 + (lane & 7)) * M::KROW + (lane >> 4) * 16 : lane * M::KROW);
      if (HD == 128) {
#pragma unroll
        for (int kk = 0; kk < AC_POS / 16; kk++) {
          uint32_t p4[4], v4[4];
          ldsm4(p4, pa + kk * 32);
          ldsm4t(v4, va + kk * 16 * M::KROW);
          mma_f16_rn(acc[0], p4, v4[0], v4[1]);
          mma_f16_rn(acc[HD / 64 - 1], p4, v4[2], v4[3]);
        }
      } else {
#pragma unroll
        for (int kk = 0; kk < AC_POS / 32; kk++) {
          uint32_t p4[4], v4[4];
          ldsm4t(v4, va + kk * 32 * M::KROW);
          ldsm4(p4, pa + kk * 64);
          mma_f16_rn(acc[0], p4, v4[0], v4[1]);
          ldsm4(p4, pa + kk * 64 + 32);
          mma_f16_rn(acc[0], p4, v4[2], v4[3]);
        }
      }
      }
    }
    if (ch + 2 < c1) __syncthreads();                                // everybody is done with the values
    fetch(ch + 2, vc, M::V, M::VROW, pos);
  }
  asm volatile("cp.async.wait_group 0;" ::: "memory");
#pragma unroll
  for (int j = 0; j < HD / 64; j++)
    *reinterpret_cast<float2*>(s_o + g * HD + warp * (HD / 8) + j * 8 + 2 * t) = make_float2(acc[j][0] + acc[j][2], acc[j][1] + acc[j][3]);
  cluster_sync();
  // merge: the (head, 32 dims) units are dealt over the cluster's CTAs, one warp each
  bool arrived = false;
  for (int u = warp * CL + rank; u < n_rep * (HD / 32); u += AC_THREADS / 32 * CL) {
    const int h = u / (HD / 32), d = (u - h * (HD / 32)) * 32 + lane;
    const uint32_t st = base + M::ST + h * 4, oa = base + M::O + (h * HD + d) * 4;
    float o[CL];
#pragma unroll
    for (int s = 0; s < CL; s++) o[s] = ld_cluster(oa, s);
    const float m = lane < CL ? ld_cluster(st, lane) : -INFINITY, l = lane < CL ? ld_cluster(st + 32, lane) : 0.f;
    if (CL > 1) { cluster_arrive(); arrived = true; }                // the last remote load
    const float w = __expf(m - warp_max(m));                         // 0 for CTAs without positions
    const float den = warp_sum(w * l);
    float v = 0.f;
#pragma unroll
    for (int s = 0; s < CL; s++) v = fmaf(__shfl_sync(0xffffffffu, w, s), o[s], v);
    v /= den;
    a.out[(size_t)(kvh * n_rep + h) * HD + d] = v;
    if (a.xq_out) quant_block_32x1(v, lane, (kvh * n_rep + h) * (HD / 32) + (d >> 5), XqDst(a.xq_out, a.n_heads));      // head_dim 128: one group per head
    if (CL > 1) break;                                               // one unit per warp at most
  }
  if (CL > 1) {                                                      // nobody leaves while its partial results are being read
    if (!arrived) cluster_arrive();
    cluster_wait();
  }
}

// ---------------------------------------------------------------------------
// arg-max with the lowest index winning ties, then tokens[pos+1] = it and pos += 1.
// scratch: float val[ARGMAX_CTAS], int idx[ARGMAX_CTAS], uint counter.
constexpr int ARGMAX_CTAS = 128;
constexpr int ARGMAX_THREADS = 256;
constexpr size_t ARGMAX_SCRATCH = ARGMAX_CTAS * (sizeof(float) + sizeof(int)) + sizeof(unsigned);

__device__ __forceinline__ void argmax_combine(float& v, int& i, float ov, int oi) {
  if (ov > v || (ov == v && oi < i)) { v = ov; i = oi; }
}

__global__ void __launch_bounds__(ARGMAX_THREADS) argmax_kernel(const float* __restrict__ logits, int n, int32_t* tokens, int32_t* pos,
                                                                int max_context, int token_stride, unsigned char* scratch, int32_t* mirror) {
  __shared__ float wv[ARGMAX_THREADS / 32];
  __shared__ int wi[ARGMAX_THREADS / 32];
  __shared__ int s_last;
  // blockIdx.y: the sequence
  logits += (size_t)blockIdx.y * n; tokens += (size_t)blockIdx.y * token_stride; pos += blockIdx.y;
  float* sval = reinterpret_cast<float*>(scratch + (size_t)blockIdx.y * ARGMAX_SCRATCH);
  int* sidx = reinterpret_cast<int*>(sval + ARGMAX_CTAS);
  unsigned* counter = reinterpret_cast<unsigned*>(sidx + ARGMAX_CTAS);
  pdl_launch_dependents();
  pdl_wait();
  float v = -INFINITY; int idx = 0x7fffffff;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) argmax_combine(v, idx, logits[i], i);
  auto block_reduce = [&]() {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      float ov = __shfl_xor_sync(0xffffffffu, v, o); int oi = __shfl_xor_sync(0xffffffffu, idx, o);
      argmax_combine(v, idx, ov, oi);
    }
    if ((threadIdx.x & 31) == 0) { wv[threadIdx.x >> 5] = v; wi[threadIdx.x >> 5] = idx; }
    __syncthreads();
    if (threadIdx.x < 32) {
      v = threadIdx.x < ARGMAX_THREADS / 32 ? wv[threadIdx.x] : -INFINITY;
      idx = threadIdx.x < ARGMAX_THREADS / 32 ? wi[threadIdx.x] : 0x7fffffff;
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) {
        float ov = __shfl_xor_sync(0xffffffffu, v, o); int oi = __shfl_xor_sync(0xffffffffu, idx, o);
        argmax_combine(v, idx, ov, oi);
      }
    }
  };
  block_reduce();
  if (threadIdx.x == 0) {
    sval[blockIdx.x] = v; sidx[blockIdx.x] = idx;
    __threadfence();
    unsigned prev = atomicAdd(counter, 1u);
    s_last = (prev == gridDim.x - 1);
    if (s_last) *counter = 0;
  }
  __syncthreads();
  if (!s_last) return;
  __threadfence();
  v = -INFINITY; idx = 0x7fffffff;
  for (int i = threadIdx.x; i < (int)gridDim.x; i += blockDim.x) argmax_combine(v, idx, __ldcg(sval + i), __ldcg(sidx + i));
  __syncthreads();
  block_reduce();
  if (threadIdx.x == 0) {
    const int p = *pos;
    if (p < 0 || p >= max_context) atomicExch(&g_decode_status, 2);      // tokens[max_context] is the last entry
    else {
      const int tok = idx == 0x7fffffff ? 0 : idx;
      tokens[p + 1] = tok; *pos = p + 1;
      if (mirror) { __threadfence_system(); *reinterpret_cast<volatile int32_t*>(mirror + blockIdx.y) = tok; }      // the host is waiting for it
    }
  }
}

}  // namespace

int b200q_decode_status_take(int* status) {
  int zero = 0;
  B200Q_CHECK_CUDA(cudaMemcpyFromSymbol(status, g_decode_status, sizeof(int)));
  B200Q_CHECK_CUDA(cudaMemcpyToSymbol(g_decode_status, &zero, sizeof(int)));
  return B200Q_OK;
}

extern "C" int b200q_embed(const void* table, const int32_t* tokens, const int32_t* pos, float* x, int dim, int vocab, int max_context, void* xq_out,
                           const void* xq_norm_weight, float* ss_out, int flags, void* stream) {
  if (!table || !tokens || !pos || !x || dim <= 0 || vocab <= 0 || max_context <= 0) return B200Q_ERR_BAD_ARG;
  if ((uintptr_t)xq_out & 15) return B200Q_ERR_MISALIGNED;
  if (xq_out && dim % 32) return B200Q_ERR_BAD_SHAPE;
  B200Q_CHECK_CUDA(launch_k(embed_kernel, dim3(ceil_div(dim, 256)), dim3(256), 0, (cudaStream_t)stream, (flags & B200Q_FLAG_PDL) != 0,
                            (const __half*)table, tokens, pos, x, dim, vocab, max_context, xq_out, (const __half*)xq_norm_weight, ss_out));
  return B200Q_OK;
}

extern "C" int b200q_advance(int32_t* pos, int max_context, int flags, void* stream) {
  if (!pos || max_context <= 0) return B200Q_ERR_BAD_ARG;
  B200Q_CHECK_CUDA(launch_k(advance_kernel, dim3(1), dim3(32), 0, (cudaStream_t)stream, (flags & B200Q_FLAG_PDL) != 0, pos, max_context));
  return B200Q_OK;
}

extern "C" int b200q_attn_min_split(int max_context) { return max_context <= 0 ? 0 : ceil_div(max_context, ATTN_CHUNK); }

extern "C" size_t b200q_attn_scratch_bytes(int n_heads, int n_kv_heads, int head_dim, int n_split) {
  if (n_heads <= 0 || n_kv_heads <= 0 || head_dim <= 0 || n_split <= 0) return 0;
  return ((size_t)n_heads * n_split * (head_dim + 4)) * sizeof(float) + (size_t)n_kv_heads * sizeof(unsigned);
}

// Argument checks shared by both attention entry points (`scratch` is checked by the caller that needs it).
static int attn_validate(const b200q_attn_args* a) {
  if (!a || !a->qkv || !a->k_cache || !a->v_cache || !a->rope || !a->pos || !a->out) return B200Q_ERR_BAD_ARG;
  if (a->n_heads <= 0 || a->n_kv_heads <= 0 || a->n_heads % a->n_kv_heads || a->n_split <= 0 || a->max_context <= 0) return B200Q_ERR_BAD_ARG;
  if (a->head_dim <= 0 || a->head_dim > MAX_HD || a->head_dim % 8 || a->n_heads / a->n_kv_heads > MAX_REP) return B200Q_ERR_BAD_SHAPE;
  if (a->rope_dim < 0 || a->rope_dim > a->head_dim || a->rope_dim % 2) return B200Q_ERR_BAD_SHAPE;
  if (a->kv_dtype != B200Q_F16 && a->kv_dtype != B200Q_F32) return B200Q_ERR_BAD_ARG;
  if (a->xq_out && (a->head_dim != 128 || ((uintptr_t)a->xq_out & 15))) return B200Q_ERR_BAD_SHAPE;   // one 128-wide group per head
  if (((uintptr_t)a->k_cache | (uintptr_t)a->v_cache | (uintptr_t)a->qkv | (uintptr_t)a->out) & 15) return B200Q_ERR_MISALIGNED;
  if ((int64_t)a->n_split * ATTN_CHUNK < a->max_context) return B200Q_ERR_BAD_SHAPE;   // the slices must cover the whole cache
  return B200Q_OK;
}

extern "C" size_t b200q_attn_seq_scratch_stride(int n_heads, int n_kv_heads, int head_dim, int n_split) {
  return (b200q_attn_scratch_bytes(n_heads, n_kv_heads, head_dim, n_split) + 255) & ~(size_t)255;
}

template <int HD, int CL, typename KV>
static int launch_attn_cluster(const b200q_attn_args* a, const SeqStride& sq, int n_seqs, bool pdl, cudaStream_t stream, int* max_clusters = nullptr) {
  auto kern = attn_cluster_kernel<HD, CL, KV>;
  static PerDeviceFlag attr_set;
  const int dev = b200q_current_device();
  if (dev < 0) return B200Q_ERR_CUDA;
  if (!attr_set.test(dev)) {
    B200Q_CHECK_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (AcSmem<HD, KV>::TOTAL)));
    if (CL > 8) B200Q_CHECK_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeNonPortableClusterSizeAllowed, 1));
    attr_set.set(dev);
  }
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(a->n_kv_heads, CL, n_seqs); cfg.blockDim = dim3(AC_THREADS); cfg.dynamicSmemBytes = (AcSmem<HD, KV>::TOTAL); cfg.stream = stream;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = 1; attr[0].val.clusterDim.y = CL; attr[0].val.clusterDim.z = 1;
  attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[1].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = CL > 1 ? attr : attr + 1; cfg.numAttrs = (CL > 1) + pdl;
  if (max_clusters) {                                                // how many clusters run at once (0: not even one)
    cfg.numAttrs = 1;
    B200Q_CHECK_CUDA(cudaOccupancyMaxActiveClusters(max_clusters, kern, &cfg));
    return B200Q_OK;
  }
  B200Q_CHECK_CUDA(cudaLaunchKernelEx(&cfg, kern, *a, sq));
  return B200Q_OK;
}

// Clusters of 16 CTAs where the device runs all KV heads' clusters at once (14 of them on B200), of 8 (portable) otherwise: with few KV heads the
// cached rows stream through twice the SMs (4 heads, position 3507: 17.9 -> 12.6 us per block); at short contexts both take the same time.
template <int HD, typename KV>
static int attn_cluster(const b200q_attn_args* a, const SeqStride& sq, int n_seqs, bool pdl, cudaStream_t stream) {
  // A cache of one chunk (a model built for at most 64 positions): one CTA does it all, the others of a cluster would only wait.  16 tokens of a 3-block 512-wide model
  // 955 us with clusters, 885 so; 8 tokens of a batch of 11 on 14 640-wide blocks 10303 us, 8223 so.  Longer caches always take clusters: the position that would
  // decide is on the device.
  if (a->max_context <= AC_POS) return launch_attn_cluster<HD, 1, KV>(a, sq, n_seqs, pdl, stream);
  static std::atomic<int> wide[B200Q_MAX_DEVICES];                   // clusters of 16 that run at once, plus one; 0: not asked yet
  const int dev = b200q_current_device();
  if (dev < 0) return B200Q_ERR_CUDA;
  int w = wide[dev].load(std::memory_order_relaxed);
  if (w == 0) {
    int n = 0;
    if (launch_attn_cluster<HD, 16, KV>(a, sq, n_seqs, pdl, stream, &n) != B200Q_OK) n = 0;
    w = n + 1;
    wide[dev].store(w, std::memory_order_relaxed);
  }
  return a->n_kv_heads * n_seqs < w ? launch_attn_cluster<HD, 16, KV>(a, sq, n_seqs, pdl, stream) : launch_attn_cluster<HD, 8, KV>(a, sq, n_seqs, pdl, stream);
}

static int attn_decode_launch(const b200q_attn_args* a, int n_seqs, void* stream) {
  const int rc = attn_validate(a);
  if (rc != B200Q_OK) return rc;
  if (!a->scratch) return B200Q_ERR_BAD_ARG;
  if ((uintptr_t)a->scratch & 15) return B200Q_ERR_MISALIGNED;
  int n_rep = a->n_heads / a->n_kv_heads;
  const int ws = 2 * n_rep <= MAX_REP ? 2 : 1;              // warps per head
  dim3 grid(a->n_kv_heads, a->n_split, n_seqs), block(ws * n_rep * 32);
  SeqStride sq = {};
  if (n_seqs > 1) {
    sq.qkv = (size_t)(a->n_heads + 2 * a->n_kv_heads) * a->head_dim; sq.cache = (size_t)a->n_kv_heads * a->max_context * a->head_dim;
    sq.out = (size_t)a->n_heads * a->head_dim; sq.pos = 1;
    sq.scratch_bytes = b200q_attn_seq_scratch_stride(a->n_heads, a->n_kv_heads, a->head_dim, a->n_split);
  }
  bool pdl = (a->flags & B200Q_FLAG_PDL) != 0;
  if (a->head_dim == 64 || a->head_dim == 128) {
    cudaStream_t st = (cudaStream_t)stream;
    if (a->kv_dtype == B200Q_F16) return a->head_dim == 128 ? attn_cluster<128, __half>(a, sq, n_seqs, pdl, st) : attn_cluster<64, __half>(a, sq, n_seqs, pdl, st);
    return a->head_dim == 128 ? attn_cluster<128, float>(a, sq, n_seqs, pdl, st) : attn_cluster<64, float>(a, sq, n_seqs, pdl, st);
  }
  const int esz = a->kv_dtype == B200Q_F16 ? 2 : 4, vec = 16 / esz;
  size_t smem = (size_t)2 * ATTN_CHUNK * (a->head_dim + vec) * esz + (size_t)n_rep * (a->head_dim + ATTN_CHUNK + a->head_dim + 4) * sizeof(float);
  static PerDeviceFlag attr_set;
  const int dev = b200q_current_device();
  if (dev < 0) return B200Q_ERR_CUDA;
  if (!attr_set.test(dev)) {
    B200Q_CHECK_CUDA(cudaFuncSetAttribute(attn_decode_kernel<float>, cudaFuncAttributeMaxDynamicSharedMemorySize, 96 * 1024));
    B200Q_CHECK_CUDA(cudaFuncSetAttribute(attn_decode_kernel<__half>, cudaFuncAttributeMaxDynamicSharedMemorySize, 96 * 1024));
    attr_set.set(dev);
  }
#ifdef B200Q_GEMV_PROF
  static int prof_counter = 0;
  b200q_attn_args ap = *a;
  ap.flags = (ap.flags & 0xFFFF) | ((prof_counter++ & 4095) << 16);
  a = &ap;
#endif
  if (a->kv_dtype == B200Q_F16) B200Q_CHECK_CUDA(launch_k(attn_decode_kernel<__half>, grid, block, smem, (cudaStream_t)stream, pdl, *a, sq));
  else B200Q_CHECK_CUDA(launch_k(attn_decode_kernel<float>, grid, block, smem, (cudaStream_t)stream, pdl, *a, sq));
  return B200Q_OK;
}

extern "C" int b200q_attn_decode(const b200q_attn_args* a, void* stream) { return attn_decode_launch(a, 1, stream); }

extern "C" int b200q_attn_decode_seqs(const b200q_attn_args* a, int n_seqs, void* stream) {
  if (n_seqs <= 0 || (a && a->xq_out)) return B200Q_ERR_BAD_ARG;
  return attn_decode_launch(a, n_seqs, stream);
}

extern "C" size_t b200q_argmax_scratch_bytes(void) { return ARGMAX_SCRATCH; }

extern "C" int b200q_argmax_advance_seqs(const float* logits, int n, int32_t* tokens, int token_stride, int32_t* pos, int max_context, void* scratch, int n_seqs,
                                         int32_t* mirror, int flags, void* stream) {
  if (!logits || !tokens || !pos || !scratch || n <= 0 || max_context <= 0 || n_seqs <= 0 || n_seqs > 65535 || token_stride < 0) return B200Q_ERR_BAD_ARG;
  int grid = ceil_div(n, ARGMAX_THREADS); if (grid > ARGMAX_CTAS) grid = ARGMAX_CTAS;
  B200Q_CHECK_CUDA(launch_k(argmax_kernel, dim3(grid, n_seqs), dim3(ARGMAX_THREADS), 0, (cudaStream_t)stream, (flags & B200Q_FLAG_PDL) != 0,
                            logits, n, tokens, pos, max_context, token_stride, (unsigned char*)scratch, mirror));
  return B200Q_OK;
}
extern "C" int b200q_argmax_advance(const float* logits, int n, int32_t* tokens, int32_t* pos, int max_context, void* scratch, int flags, void* stream) {
  return b200q_argmax_advance_seqs(logits, n, tokens, 0, pos, max_context, scratch, 1, nullptr, flags, stream);
}

// ---------------------------------------------------------------------------
// Attention for callers that may not allocate device memory.
//
// Some hosts of this library hand out device memory themselves and forbid anything else from doing so: a serving loop
// that froze its memory pool after warm-up, an engine whose planner owns one arena and replays captured work, or code
// running while a stream is being captured (the CUDA allocator calls are illegal there).  Such a caller cannot provide
// the scratch buffer b200q_attn_decode needs unless it planned for it.  This variant brings its own: a fixed array that
// is part of the library image, so every GPU that loads the library holds these bytes until the process exits.
constexpr size_t ATTN_STATIC_SCRATCH_BYTES = (size_t)2 << 20;     // 2 MiB: e.g. 64 heads x 62 slices (3968 positions) of head_dim 128
static __device__ __align__(256) unsigned char g_attn_static_scratch[ATTN_STATIC_SCRATCH_BYTES];

constexpr int MAX_DEVICES = B200Q_MAX_DEVICES;
static void* g_attn_static_ptr[MAX_DEVICES];   // device address of the array on each device, filled on first use

extern "C" size_t b200q_attn_decode_static_capacity(void) { return ATTN_STATIC_SCRATCH_BYTES; }

extern "C" int b200q_attn_decode_static(const b200q_attn_args* a, void* stream) {
  if (!a) return B200Q_ERR_BAD_ARG;
  const size_t need = b200q_attn_scratch_bytes(a->n_heads, a->n_kv_heads, a->head_dim, a->n_split);
  if (need == 0) return B200Q_ERR_BAD_ARG;
  if (need > ATTN_STATIC_SCRATCH_BYTES) return B200Q_ERR_TOO_LARGE;
  const int rc = attn_validate(a);      // before anything is put on the stream
  if (rc != B200Q_OK) return rc;   // heads x slices x (head_dim + 4) floats must fit the built-in array
  int dev = -1;
  B200Q_CHECK_CUDA(cudaGetDevice(&dev));
  if (dev < 0 || dev >= MAX_DEVICES) return B200Q_ERR_TOO_LARGE;
  if (!g_attn_static_ptr[dev]) {
    // In host code the array's name is only a handle; the kernel needs the address the array has on THIS device.
    void* p = nullptr;
    B200Q_CHECK_CUDA(cudaGetSymbolAddress(&p, g_attn_static_scratch));
    g_attn_static_ptr[dev] = p;
  }
  // The arrival counters sit behind the partial results, at an offset that depends on the geometry, and the array keeps
  // whatever the last call left there: zero them (stream-ordered, no allocation) before the kernel counts arrivals.
  unsigned char* base = static_cast<unsigned char*>(g_attn_static_ptr[dev]);
  const size_t counters_at = need - (size_t)a->n_kv_heads * sizeof(unsigned);
  B200Q_CHECK_CUDA(cudaMemsetAsync(base + counters_at, 0, (size_t)a->n_kv_heads * sizeof(unsigned), (cudaStream_t)stream));
  b200q_attn_args b = *a;
  b.scratch = base;
  b.flags &= ~B200Q_FLAG_PDL;   // the memset in front is not a kernel: launch the kernel fully ordered behind it
  return b200q_attn_decode(&b, stream);
}
