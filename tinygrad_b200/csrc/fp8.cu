// Per-tensor FP8 (E4M3) linear: `quantize_to_fp8` and the scaling behind the product of `FP8Linear.__call__`
// (extra/fp8/fp8_linear.py:4-16,43-63): scale = 448 / (max|x| + 1e-8) over the WHOLE tensor, q = e4m3(clamp(x * scale, +-448)), the
// returned factor is 1 / scale; y = (x_q . w_q^T, fp32) * w_factor * x_factor + bias, cast to the activation dtype.
// The contraction itself is the grouped tcgen05 GEMM with unit block scales and fp32 output (b200q_grouped_mxfp8_gemm_f32).
#include "common.cuh"
#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <cuda_fp8.h>
#include <cooperative_groups.h>

namespace {

template <typename T> __device__ __forceinline__ float ldf(const T* p, int64_t i);
template <> __device__ __forceinline__ float ldf<float>(const float* p, int64_t i) { return p[i]; }
template <> __device__ __forceinline__ float ldf<__half>(const __half* p, int64_t i) { return __half2float(p[i]); }
template <> __device__ __forceinline__ float ldf<__nv_bfloat16>(const __nv_bfloat16* p, int64_t i) { return __bfloat162float(p[i]); }

// eight consecutive values; base pointers are at least 16-byte aligned where VEC is used
template <typename T> __device__ __forceinline__ void ld8(const T* p, int64_t i, float (&v)[8]);
template <> __device__ __forceinline__ void ld8<float>(const float* p, int64_t i, float (&v)[8]) {
  const float4 a = *reinterpret_cast<const float4*>(p + i), b = *reinterpret_cast<const float4*>(p + i + 4);
  v[0] = a.x; v[1] = a.y; v[2] = a.z; v[3] = a.w; v[4] = b.x; v[5] = b.y; v[6] = b.z; v[7] = b.w;
}
template <> __device__ __forceinline__ void ld8<__half>(const __half* p, int64_t i, float (&v)[8]) {
  const uint4 r = *reinterpret_cast<const uint4*>(p + i);
  const __half2* h = reinterpret_cast<const __half2*>(&r);
#pragma unroll
  for (int q = 0; q < 4; q++) { const float2 f = __half22float2(h[q]); v[2 * q] = f.x; v[2 * q + 1] = f.y; }
}
template <> __device__ __forceinline__ void ld8<__nv_bfloat16>(const __nv_bfloat16* p, int64_t i, float (&v)[8]) {
  const uint4 r = *reinterpret_cast<const uint4*>(p + i);
  const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&r);
#pragma unroll
  for (int q = 0; q < 4; q++) { const float2 f = __bfloat1622float2(h[q]); v[2 * q] = f.x; v[2 * q + 1] = f.y; }
}

// Both passes are bound by memory and, for a few rows, by latency: eight values per thread and load (16 or 32 bytes) instead of one.
// The maximum goes out as one partial value per block, which the quantising kernel folds: no cleared word, no atomics, one launch less.
// (|x| is non-negative; NaN inputs are not expected.)
constexpr int Q_THREADS = 256, MAX_PARTS = 592;

template <typename T>
__device__ __forceinline__ float block_absmax(const T* __restrict__ x, int64_t n, bool vec) {
  __shared__ float red[Q_THREADS / 32];
  float m = 0.f;
  const int64_t t = (int64_t)blockIdx.x * Q_THREADS + threadIdx.x, step = (int64_t)gridDim.x * Q_THREADS, n8 = vec ? n / 8 : 0;
  for (int64_t i = t; i < n8; i += step) {
    float v[8];
    ld8<T>(x, i * 8, v);
#pragma unroll
    for (int j = 0; j < 8; j++) m = fmaxf(m, fabsf(v[j]));
  }
  for (int64_t i = n8 * 8 + t; i < n; i += step) m = fmaxf(m, fabsf(ldf<T>(x, i)));
  m = warp_max(m);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = m;
  __syncthreads();
#pragma unroll
  for (int w = 0; w < Q_THREADS / 32; w++) m = fmaxf(m, red[w]);
  return m;
}
template <typename T>
__global__ void __launch_bounds__(Q_THREADS) fp8_absmax_kernel(const T* __restrict__ x, int64_t n, unsigned* __restrict__ amax_bits, int vec) {
  const float m = block_absmax<T>(x, n, vec);
  if (threadIdx.x == 0) atomicMax(amax_bits, __float_as_uint(m));
}
template <typename T>
__global__ void __launch_bounds__(Q_THREADS) fp8_absmax_parts_kernel(const T* __restrict__ x, int64_t n, float* __restrict__ parts, int vec) {
  pdl_wait();
  pdl_launch_dependents();
  const float m = block_absmax<T>(x, n, vec);
  if (threadIdx.x == 0) parts[blockIdx.x] = m;
}

struct Scale {      // of a tensor whose largest magnitude is m
  float d, scale;
  __device__ __forceinline__ explicit Scale(float m) { d = __fadd_rn(m, 1e-8f); scale = __fdiv_rn(448.f, d); }
  __device__ __forceinline__ float factor() const { return __fmul_rn(d, 1.f / 448.f); }      // the reference's simplified (448 / d).reciprocal()
  __device__ __forceinline__ uint32_t code(float f) const { return (uint32_t)__nv_cvt_float_to_fp8(fminf(fmaxf(__fmul_rn(f, scale), -448.f), 448.f), __NV_SATFINITE, __NV_E4M3); }
  __device__ __forceinline__ uint2 code8(const float (&v)[8]) const {
    return make_uint2(code(v[0]) | code(v[1]) << 8 | code(v[2]) << 16 | code(v[3]) << 24, code(v[4]) | code(v[5]) << 8 | code(v[6]) << 16 | code(v[7]) << 24);
  }
};

// Both passes in one launch, as long as the tensor fits the registers of a CTA of 1024 threads per SM, HOLD pieces of eight values a thread (4.8 million values on 148 SMs): read once,
// the partial maxima meet behind a grid barrier (cooperative launch; none where one CTA has it all), the codes come from the registers.  The two launches read the tensor
// twice and stand behind one another.  FP8 linear, us a call, two launches / so: 1 x 4096 -> 4096 20.9 / 19.4, 1 x 2048 -> 6144 14.7 / 12.5, 500 x 4096 23.2 / 21.7, 1000 x 4096
// 33.6 / 31.6, 1000 x 2048 33.0 / 31.5; between one CTA and WHOLE_MIN values the barrier costs what the launch did: 500 x 1024 15.7 / 16.2, 20 x 6144 22.9 / 24.3.
// n a multiple of 8, x 16-byte aligned.
constexpr int WHOLE_THREADS = 1024, HOLD = 4;
constexpr int64_t WHOLE_MIN = 1 << 20;
template <typename T>
__global__ void __launch_bounds__(WHOLE_THREADS, 1) fp8_quantize_whole_kernel(const T* __restrict__ x, int64_t n8, float* __restrict__ parts, uint8_t* __restrict__ q,
                                                                             float* __restrict__ factor) {
  __shared__ float red[WHOLE_THREADS / 32];
  const int64_t t = (int64_t)blockIdx.x * WHOLE_THREADS + threadIdx.x, step = (int64_t)gridDim.x * WHOLE_THREADS;
  float v[HOLD][8], m = 0.f;
#pragma unroll
  for (int i = 0; i < HOLD; i++) {
#pragma unroll
    for (int j = 0; j < 8; j++) v[i][j] = 0.f;
    if (t + i * step < n8) ld8<T>(x, (t + i * step) * 8, v[i]);
  }
  pdl_launch_dependents();
#pragma unroll
  for (int i = 0; i < HOLD; i++)
#pragma unroll
    for (int j = 0; j < 8; j++) m = fmaxf(m, fabsf(v[i][j]));
  auto over_block = [&]() {
    m = warp_max(m);
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = m;
    __syncthreads();
    m = warp_max(red[threadIdx.x & 31]);
  };
  over_block();
  if (gridDim.x > 1) {
    if (threadIdx.x == 0) parts[blockIdx.x] = m;
    cooperative_groups::this_grid().sync();
    m = 0.f;
    for (int i = threadIdx.x; i < (int)gridDim.x; i += WHOLE_THREADS) m = fmaxf(m, __ldcg(parts + i));
    over_block();
  }
  const Scale sc(m);
  if (t == 0) *factor = sc.factor();
#pragma unroll
  for (int i = 0; i < HOLD; i++) if (t + i * step < n8) reinterpret_cast<uint2*>(q)[t + i * step] = sc.code8(v[i]);
}

// amax: n_parts partial maxima (or the one maximum)
template <typename T>
__global__ void __launch_bounds__(Q_THREADS) fp8_quantize_kernel(const T* __restrict__ x, int64_t n, const float* __restrict__ amax, int n_parts,
                                                                 uint8_t* __restrict__ q, float* __restrict__ factor, int vec) {
  __shared__ float red[Q_THREADS / 32];
  pdl_wait();
  pdl_launch_dependents();
  float m = 0.f;
  for (int i = threadIdx.x; i < n_parts; i += Q_THREADS) m = fmaxf(m, amax[i]);
  m = warp_max(m);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = m;
  __syncthreads();
#pragma unroll
  for (int w = 0; w < Q_THREADS / 32; w++) m = fmaxf(m, red[w]);
  const Scale sc(m);
  if (blockIdx.x == 0 && threadIdx.x == 0) *factor = sc.factor();
  const int64_t t = (int64_t)blockIdx.x * Q_THREADS + threadIdx.x, step = (int64_t)gridDim.x * Q_THREADS, n8 = vec ? n / 8 : 0;
  for (int64_t i = t; i < n8; i += step) {
    float v[8];
    ld8<T>(x, i * 8, v);
    reinterpret_cast<uint2*>(q)[i] = sc.code8(v);
  }
  for (int64_t i = n8 * 8 + t; i < n; i += step) q[i] = (uint8_t)sc.code(ldf<T>(x, i));
}

template <typename T> __device__ __forceinline__ void stf(T* p, int64_t i, float v);
template <> __device__ __forceinline__ void stf<float>(float* p, int64_t i, float v) { p[i] = v; }
template <> __device__ __forceinline__ void stf<__half>(__half* p, int64_t i, float v) { p[i] = __float2half_rn(v); }
template <> __device__ __forceinline__ void stf<__nv_bfloat16>(__nv_bfloat16* p, int64_t i, float v) { p[i] = __float2bfloat16_rn(v); }

template <typename T>
__global__ void fp8_scale_bias_kernel(const float* __restrict__ acc, int64_t rows, int n, const float* __restrict__ fw, const float* __restrict__ fx,
                                      const float* __restrict__ bias, T* __restrict__ y) {
  const float w = *fw, xx = *fx;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < rows * n; i += (int64_t)gridDim.x * blockDim.x) {
    float v = __fmul_rn(__fmul_rn(acc[i], w), xx);                 // y * w_scale * x_scale, in that order
    if (bias) v = __fadd_rn(v, bias[i % n]);
    stf<T>(y, i, v);
  }
}

// blocks for n values, eight per thread: up to four per SM
int quant_grid(int64_t n) {
  const int64_t b = (n / 8 + Q_THREADS - 1) / Q_THREADS, most = min(4 * b200q_sm_count(), MAX_PARTS);
  return (int)(b < 1 ? 1 : (b > most ? most : b));
}
// The launch of fp8_quantize_whole_kernel: a thread for every eight values while there are SMs for them.
template <typename T> cudaError_t launch_whole(const T* x, int64_t n, int n_sm, float* parts, void* q, float* factor, cudaStream_t st) {
  const int64_t ctas = (n / 8 + WHOLE_THREADS - 1) / WHOLE_THREADS;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)(ctas < n_sm ? ctas : n_sm)); cfg.blockDim = dim3(WHOLE_THREADS); cfg.stream = st;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeCooperative;
  attr[0].val.cooperative = 1;
  cfg.attrs = attr; cfg.numAttrs = cfg.gridDim.x > 1;
  return cudaLaunchKernelEx(&cfg, fp8_quantize_whole_kernel<T>, x, n / 8, parts, (uint8_t*)q, factor);
}
int grid_for(int64_t n) { const int64_t b = (n + 255) / 256; return (int)(b < 1 ? 1 : (b > 4096 ? 4096 : b)); }

}  // namespace

extern "C" int b200q_fp8_absmax(const void* x, int x_dtype, int64_t n, float* amax, void* stream) {
  if (!x || !amax || n <= 0) return B200Q_ERR_BAD_ARG;
  cudaStream_t st = (cudaStream_t)stream;
  B200Q_CHECK_CUDA(cudaMemsetAsync(amax, 0, sizeof(float), st));
  const int g = quant_grid(n), vec = !((uintptr_t)x & 15);
  if (x_dtype == B200Q_F32) fp8_absmax_kernel<float><<<g, Q_THREADS, 0, st>>>((const float*)x, n, (unsigned*)amax, vec);
  else if (x_dtype == B200Q_F16) fp8_absmax_kernel<__half><<<g, Q_THREADS, 0, st>>>((const __half*)x, n, (unsigned*)amax, vec);
  else if (x_dtype == B200Q_BF16) fp8_absmax_kernel<__nv_bfloat16><<<g, Q_THREADS, 0, st>>>((const __nv_bfloat16*)x, n, (unsigned*)amax, vec);
  else return B200Q_ERR_BAD_ARG;
  B200Q_CHECK_CUDA(cudaGetLastError());
  return B200Q_OK;
}

extern "C" int b200q_fp8_quantize(const void* x, int x_dtype, int64_t n, const float* amax, void* q, float* factor, void* stream) {
  if (!x || !amax || !q || !factor || n <= 0) return B200Q_ERR_BAD_ARG;
  cudaStream_t st = (cudaStream_t)stream;
  const int g = quant_grid(n), vec = !((uintptr_t)x & 15) && !((uintptr_t)q & 7);
  if (x_dtype == B200Q_F32) fp8_quantize_kernel<float><<<g, Q_THREADS, 0, st>>>((const float*)x, n, amax, 1, (uint8_t*)q, factor, vec);
  else if (x_dtype == B200Q_F16) fp8_quantize_kernel<__half><<<g, Q_THREADS, 0, st>>>((const __half*)x, n, amax, 1, (uint8_t*)q, factor, vec);
  else if (x_dtype == B200Q_BF16) fp8_quantize_kernel<__nv_bfloat16><<<g, Q_THREADS, 0, st>>>((const __nv_bfloat16*)x, n, amax, 1, (uint8_t*)q, factor, vec);
  else return B200Q_ERR_BAD_ARG;
  B200Q_CHECK_CUDA(cudaGetLastError());
  return B200Q_OK;
}

extern "C" int b200q_fp8_scale_bias(const float* acc, int64_t rows, int n, const float* factor_w, const float* factor_x, const float* bias, void* y, int y_dtype,
                                    void* stream) {
  if (!acc || !factor_w || !factor_x || !y || rows <= 0 || n <= 0) return B200Q_ERR_BAD_ARG;
  cudaStream_t st = (cudaStream_t)stream;
  const int g = grid_for(rows * n);
  if (y_dtype == B200Q_F32) fp8_scale_bias_kernel<float><<<g, 256, 0, st>>>(acc, rows, n, factor_w, factor_x, bias, (float*)y);
  else if (y_dtype == B200Q_F16) fp8_scale_bias_kernel<__half><<<g, 256, 0, st>>>(acc, rows, n, factor_w, factor_x, bias, (__half*)y);
  else if (y_dtype == B200Q_BF16) fp8_scale_bias_kernel<__nv_bfloat16><<<g, 256, 0, st>>>(acc, rows, n, factor_w, factor_x, bias, (__nv_bfloat16*)y);
  else return B200Q_ERR_BAD_ARG;
  B200Q_CHECK_CUDA(cudaGetLastError());
  return B200Q_OK;
}

// The whole call in two launches (maximum and codes, product with the factors and the bias in its epilogue) or, where one cannot have the tensor in registers, three; the
// result in a pool block.
extern "C" int b200q_fp8_linear(const b200q_fp8_linear_desc* l, const void* x, int dtype, int m, void** y, void* stream) {
  if (!l || !y || m <= 0 || !x || (dtype != B200Q_F32 && dtype != B200Q_F16)) return B200Q_ERR_BAD_ARG;
  if (!l->w_q || !l->w_factor || !l->x_q || !l->off || !l->parts || !l->factor || m > l->rows_max) return B200Q_ERR_BAD_ARG;
  if (l->n_out <= 0 || l->n_out % 256 || l->n_in <= 0 || l->n_in % 128) return B200Q_ERR_BAD_SHAPE;
  if ((uintptr_t)l->bias & 15) return B200Q_ERR_MISALIGNED;      // read 16 bytes at a time
  cudaStream_t st = (cudaStream_t)stream;
  int rc = b200q_pool_alloc(y, (size_t)m * l->n_out * (dtype == B200Q_F32 ? 4 : 2), stream);
  if (rc != B200Q_OK) return rc;
  const int64_t n = (int64_t)m * l->n_in;
  const int g = quant_grid(n), vec = !((uintptr_t)x & 15), n_sm = b200q_sm_count();
  cudaError_t e;
  if (vec && n_sm > 0 && n_sm <= MAX_PARTS && (n <= WHOLE_THREADS * 8 || n >= WHOLE_MIN) && n <= (int64_t)n_sm * WHOLE_THREADS * HOLD * 8) {
    e = dtype == B200Q_F32 ? launch_whole((const float*)x, n, n_sm, l->parts, l->x_q, l->factor, st) : launch_whole((const __half*)x, n, n_sm, l->parts, l->x_q, l->factor, st);
  } else {
    e = dtype == B200Q_F32 ? launch_k(fp8_absmax_parts_kernel<float>, dim3(g), dim3(Q_THREADS), 0, st, false, (const float*)x, n, l->parts, vec)
                           : launch_k(fp8_absmax_parts_kernel<__half>, dim3(g), dim3(Q_THREADS), 0, st, false, (const __half*)x, n, l->parts, vec);
    if (e == cudaSuccess)
      e = dtype == B200Q_F32 ? launch_k(fp8_quantize_kernel<float>, dim3(g), dim3(Q_THREADS), 0, st, true, (const float*)x, n, (const float*)l->parts, g, (uint8_t*)l->x_q,
                                        l->factor, vec)
                             : launch_k(fp8_quantize_kernel<__half>, dim3(g), dim3(Q_THREADS), 0, st, true, (const __half*)x, n, (const float*)l->parts, g, (uint8_t*)l->x_q,
                                        l->factor, vec);
  }
  if (e != cudaSuccess) { b200q_set_cuda_error(e); rc = B200Q_ERR_CUDA; }
  else rc = b200q_mx_gemm_scaled(l->x_q, l->w_q, l->off, l->rows_max, l->n_out, l->n_in, *y, dtype, m, l->w_factor, l->factor, l->bias, st);
  if (rc != B200Q_OK) { b200q_pool_free(*y); *y = nullptr; }
  return rc;
}
