// One token's way to its experts (tinygrad/llm/model.py:110-124) in one launch: RMSNorm, router logits, the choice with its tables, and the normed row's MXFP8 codes in the
// chosen experts' groups.  As four launches (rmsnorm_rows, dense_gemv, route_one, quantize_mxfp8: 11 us a block of a one-token step) each is one CTA's work behind a launch's
// latency.  Here a cluster of eight CTAs shares the experts' logits; every CTA hears all of them, chooses for itself and quantises an eighth of the row.
// Every value is what those kernels make of it, bit for bit (sums in their order): the choice and the E4M3 codes turn a last-bit difference into a visible one.
// What bounds it is latency: a warp's first router rows are in registers before the wait for the row.
#include "common.cuh"
#include "mxq.cuh"
#include "moe_route.cuh"
#include <cuda_bf16.h>
#include <cuda_fp8.h>

namespace {

constexpr int RT_CTAS = 8, RT_THREADS = 256, RT_WARPS = RT_THREADS / 32, MAX_EXPERTS = 256, MAX_K = 32, MAX_DIM = 8192, GROUP_ROWS = 256;

// eight values of a router row
__device__ __forceinline__ void router8(const float* p, float (&v)[8]) {
  const uint4 a = ldg_stream(reinterpret_cast<const uint4*>(p)), b = ldg_stream(reinterpret_cast<const uint4*>(p) + 1);
  const uint32_t u[8] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w};
#pragma unroll
  for (int i = 0; i < 8; i++) v[i] = __uint_as_float(u[i]);
}
__device__ __forceinline__ void router8(const __half* p, float (&v)[8]) {
  const uint4 u = ldg_stream(reinterpret_cast<const uint4*>(p));
  const __half2* h = reinterpret_cast<const __half2*>(&u);
#pragma unroll
  for (int i = 0; i < 4; i++) { const float2 f = __half22float2(h[i]); v[2 * i] = f.x; v[2 * i + 1] = f.y; }
}

struct RouterParams {
  const float* x;
  const __half* norm_w;
  const void* router;
  float eps;
  int dim, n_experts, k;
  RouteRule rule;
  int32_t *topi, *dest_row, *off, *ends;
  float *weights, *xn;
  uint8_t *a_q, *a_e8;
};

// EPL as in route_token.  dim % 256 == 0.  Shared memory: the normed row.
template <typename W, int EPL>
__global__ void __launch_bounds__(RT_THREADS) moe_router_kernel(const RouterParams p) {
  constexpr int PF = 4;
  extern __shared__ __align__(16) float xs[];
  __shared__ float s_logits[MAX_EXPERTS], red[RT_WARPS], s_w[MAX_K];
  __shared__ int s_topi[MAX_K], s_dest[MAX_K];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, rank = blockIdx.x;
  const W* router = reinterpret_cast<const W*>(p.router);
  const int e0 = warp * RT_CTAS + rank;                  // a warp's experts: e0, e0 + 64 ..
  float pre[PF][8];
#pragma unroll
  for (int u = 0; u < PF; u++) if (e0 < p.n_experts && u * 256 < p.dim) router8(router + (size_t)e0 * p.dim + u * 256 + lane * 8, pre[u]);
  pdl_launch_dependents();
  cluster_sync();               // every CTA of the cluster runs: its shared memory may be written
  pdl_wait();
  for (int i = tid * 4; i < p.dim; i += RT_THREADS * 4) *reinterpret_cast<float4*>(xs + i) = *reinterpret_cast<const float4*>(p.x + i);
  __syncthreads();
  float ss = 0.f;
  for (int i = tid; i < p.dim; i += RT_THREADS) { const float v = xs[i]; ss += v * v; }
  ss = warp_sum(ss);
  if (lane == 0) red[warp] = ss;
  __syncthreads();
  float tot = 0.f;
  for (int i = 0; i < RT_WARPS; i++) tot += red[i];
  const float sc = 1.0f / sqrtf(tot / (float)p.dim + p.eps);
  for (int i = tid; i < p.dim; i += RT_THREADS) {
    const float v = xs[i] * sc * __half2float(p.norm_w[i]);
    xs[i] = v;
    if (p.xn && rank == 0) p.xn[i] = v;
  }
  __syncthreads();
#pragma unroll 1
  for (int e = e0; e < p.n_experts; e += RT_CTAS * RT_WARPS) {
    float acc = 0.f;
    auto dot = [&](const float (&v)[8], int c) {
      const float4 x0 = *reinterpret_cast<const float4*>(xs + c), x1 = *reinterpret_cast<const float4*>(xs + c + 4);
      acc += v[0] * x0.x + v[1] * x0.y + v[2] * x0.z + v[3] * x0.w + v[4] * x1.x + v[5] * x1.y + v[6] * x1.z + v[7] * x1.w;
    };
    int c = lane * 8;
    if (e == e0) {
#pragma unroll
      for (int u = 0; u < PF; u++) if (u * 256 < p.dim) dot(pre[u], c + u * 256);
      c += PF * 256;
    }
#pragma unroll 4
    for (; c < p.dim; c += 256) {
      float v[8];
      router8(router + (size_t)e * p.dim + c, v);
      dot(v, c);
    }
    acc = warp_sum(acc);
    if (lane < RT_CTAS) {
      uint32_t at;
      asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(at) : "r"((uint32_t)__cvta_generic_to_shared(s_logits + e)), "r"(lane));
      asm volatile("st.shared::cluster.f32 [%0], %1;" ::"r"(at), "f"(acc) : "memory");
    }
  }
  cluster_sync();
  if (warp == 0) {
    route_token<EPL>(p.rule, s_logits, 0, p.n_experts, p.k, s_topi, s_w, nullptr);
    __syncwarp();
    // one row in each chosen expert's group, the groups in the order of the experts
    const int mine = lane < p.k ? s_topi[lane] : 0x7fffffff;
    int before = 0;
    for (int j = 0; j < p.k; j++) before += s_topi[j] < mine;
    if (lane < p.k) s_dest[lane] = before * GROUP_ROWS;
    if (rank == 0) {
      if (lane < p.k) { p.topi[lane] = mine; p.weights[lane] = s_w[lane]; p.dest_row[lane] = before * GROUP_ROWS; }
      for (int e = lane; e <= p.n_experts; e += 32) {
        int n = 0, here = 0;
        for (int j = 0; j < p.k; j++) { n += s_topi[j] < e; here |= s_topi[j] == e; }
        p.off[e] = n * GROUP_ROWS;
        if (e < p.n_experts) p.ends[e] = n * GROUP_ROWS + here;
      }
    }
  }
  __syncthreads();
  // this CTA's blocks of the row: the values as a tensor would hold them (bf16), quantised
#pragma unroll 1
  for (int b = rank * RT_WARPS + warp; b < p.dim / 32; b += RT_CTAS * RT_WARPS) {
    const float v = __bfloat162float(__float2bfloat16_rn(xs[b * 32 + lane]));
    const uint8_t e8 = mx_scale_exponent(warp_max(fabsf(v)));
    const uint8_t q = __nv_cvt_float_to_fp8(fminf(fmaxf(v * mx_inv_scale(e8), -448.f), 448.f), __NV_SATFINITE, __NV_E4M3);
    for (int j = 0; j < p.k; j++) {
      p.a_q[(size_t)s_dest[j] * p.dim + b * 32 + lane] = q;
      if (lane == 0) p.a_e8[(size_t)s_dest[j] * (p.dim >> 5) + b] = e8;
    }
  }
}

template <typename W> int launch_router(const RouterParams& p, cudaStream_t st) {
  auto kern = p.n_experts <= 32 ? moe_router_kernel<W, 1> : p.n_experts <= 64 ? moe_router_kernel<W, 2> : moe_router_kernel<W, MAX_E_PER_LANE>;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(RT_CTAS); cfg.blockDim = dim3(RT_THREADS); cfg.dynamicSmemBytes = (size_t)p.dim * sizeof(float); cfg.stream = st;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = RT_CTAS; attr[0].val.clusterDim.y = 1; attr[0].val.clusterDim.z = 1;
  attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[1].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr; cfg.numAttrs = 2;
  B200Q_CHECK_CUDA(cudaLaunchKernelEx(&cfg, kern, p));
  return B200Q_OK;
}

}  // namespace

bool b200q_moe_router_one_takes(const b200q_moe_args* m, int router_dtype) {
  return m->d % 256 == 0 && m->d <= MAX_DIM && m->n_experts > 0 && m->n_experts <= MAX_EXPERTS && m->k > 0 && m->k <= MAX_K && m->k <= m->n_experts &&
         (router_dtype == B200Q_F32 || router_dtype == B200Q_F16);
}
int b200q_moe_router_one(const b200q_moe_args* m, const void* router, int router_dtype, const float* x, const void* norm_weight, float eps, float* xn, cudaStream_t st) {
  if (!m || !router || !x || !norm_weight || !m->topi || !m->weights || !m->dest_row || !m->off || !m->ends || !m->a_q || !m->a_e8) return B200Q_ERR_BAD_ARG;
  if (!b200q_moe_router_one_takes(m, router_dtype)) return B200Q_ERR_UNSUPPORTED;
  if (m->gating ? m->gating < GATE_SOFTMAX || m->gating > GATE_SQRT_SOFTPLUS : m->mode != 0 && m->mode != 1) return B200Q_ERR_BAD_ARG;
  if (((uintptr_t)router | (uintptr_t)x) & 15) return B200Q_ERR_MISALIGNED;
  const RouterParams p{x, (const __half*)norm_weight, router, eps, m->d, m->n_experts, m->k, RouteRule{m->mode, m->gating, m->normalize, m->scale, m->sel_bias}, m->topi,
                       m->dest_row, m->off, m->ends, m->weights, xn, (uint8_t*)m->a_q, (uint8_t*)m->a_e8};
  return router_dtype == B200Q_F32 ? launch_router<float>(p, st) : launch_router<__half>(p, st);
}
