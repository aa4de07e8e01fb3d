// One fp32 activation row times a packed Q4_0 / Q8_0 matrix, in fp32 throughout: y = W . (norm(x)) (+ bias) (+ residual), or silu(gate) . up.
//
// For Linears so small that a launch is latency and not bytes: the GEMV of gemv.cu streams any matrix through a ring, quantises the row in every CTA and hands sums
// between warps by barriers; here a CTA takes ONE row tile, its warps share the tile's K groups, and
//  * the weights a warp needs first are in registers before the wait for the previous kernel, whose tail and launch gap they cross;
//  * the row is staged as it is (times the norm weight; the RMS factor multiplies the sum): one load, one store, one block barrier, no maximum and no division;
//  * a quant becomes a float by one byte permutation (2^23 + q) and half a packed subtraction, products and sums are packed fp32 FMAs: 32 products of a block, then
//    one FMA with its scale.  2.2 instructions a weight against 0.6 of the int8 form, for matrices where neither shows.
// Nothing is rounded but the sums, where 15-bit activation codes are 4e-5 off.  512 x 512: 2.4 -> 1.7 us a launch in a chain (an empty kernel 0.84); 16 tokens of a
// 512-wide model of 3 blocks 907 -> 764 us.
#include "common.cuh"

namespace {

struct RowGemvParams {
  const uint8_t* w;
  const float* x;
  const __half *norm_w, *bias;
  const float* residual;
  float* y;
  int n_out, n_in, kgroups, epilogue;
  float eps;
};

constexpr int XB = 36;      // floats a block of 32 takes in shared memory: the four lanes of a quad read four blocks, on banks 4 apart

// two floats in a 64-bit register: the packed fp32 instructions
typedef unsigned long long f2;
__device__ __forceinline__ f2 pack2(float a, float b) { f2 r; asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b)); return r; }
__device__ __forceinline__ f2 add2(f2 a, f2 b) { f2 r; asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b)); return r; }
__device__ __forceinline__ f2 fma2(f2 a, f2 b, f2 c) { f2 r; asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c)); return r; }
__device__ __forceinline__ float sum2(f2 a, f2 b) {
  float x, y;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(x), "=f"(y) : "l"(add2(a, b)));
  return x + y;
}

// What a lane holds of a tile (16 rows x 128 columns): its block of row g and of row g + 8, and their scales.
template <int QT> struct LaneTile {
  static constexpr int Q = QT == B200Q_Q4_0 ? 1 : 2;      // 16-byte pieces of a block
  uint4 r0[Q], r1[Q];
  uint2 d;
  __device__ __forceinline__ void load(const uint8_t* tile, int lane) {
    const uint4* tp = reinterpret_cast<const uint4*>(tile);
#pragma unroll
    for (int i = 0; i < Q; i++) { r0[i] = ldg_stream(tp + 32 * i + lane); r1[i] = ldg_stream(tp + 32 * (Q + i) + lane); }
    d = ldg_stream(reinterpret_cast<const uint2*>(tile + 1024 * Q) + (lane >> 1));      // {row g: blocks t & ~1, t | 1}, {row g + 8: the same}
  }
};
// acc += four bytes of w (each q + OFF) times x[0 .. 3]
template <int OFF> __device__ __forceinline__ void mac4(uint32_t w, f2 x01, f2 x23, f2& acc0, f2& acc1) {
  const f2 off = pack2(-(8388608.f + OFF), -(8388608.f + OFF));
  auto f = [&](int k) { return __uint_as_float(__byte_perm(w, 0x4B000000u, 0x7540 + k)); };
  acc0 = fma2(add2(pack2(f(0), f(1)), off), x01, acc0);
  acc1 = fma2(add2(pack2(f(2), f(3)), off), x23, acc1);
}
// x: the lane's block of the group in shared memory
template <int QT> __device__ __forceinline__ void tile_dot(const LaneTile<QT>& w, const float* x, int t, float& a0, float& a1) {
  f2 s0 = 0, s1 = 0, u0 = 0, u1 = 0;
#pragma unroll
  for (int i = 0; i < 4; i++) {
    auto word = [](const uint4& v, int k) { return k == 0 ? v.x : k == 1 ? v.y : k == 2 ? v.z : v.w; };
    const float4 xa = *reinterpret_cast<const float4*>(x + 4 * i), xb = *reinterpret_cast<const float4*>(x + 16 + 4 * i);
    const f2 a01 = pack2(xa.x, xa.y), a23 = pack2(xa.z, xa.w), b01 = pack2(xb.x, xb.y), b23 = pack2(xb.z, xb.w);
    if constexpr (QT == B200Q_Q4_0) {      // byte i: element i | element i + 16 << 4
      const uint32_t v0 = word(w.r0[0], i), v1 = word(w.r1[0], i), M = 0x0F0F0F0Fu;
      mac4<8>(v0 & M, a01, a23, s0, s1); mac4<8>((v0 >> 4) & M, b01, b23, s0, s1);
      mac4<8>(v1 & M, a01, a23, u0, u1); mac4<8>((v1 >> 4) & M, b01, b23, u0, u1);
    } else {
      mac4<128>(word(w.r0[0], i) ^ 0x80808080u, a01, a23, s0, s1); mac4<128>(word(w.r0[1], i) ^ 0x80808080u, b01, b23, s0, s1);
      mac4<128>(word(w.r1[0], i) ^ 0x80808080u, a01, a23, u0, u1); mac4<128>(word(w.r1[1], i) ^ 0x80808080u, b01, b23, u0, u1);
    }
  }
  const __half2 h0 = *reinterpret_cast<const __half2*>(&w.d.x), h1 = *reinterpret_cast<const __half2*>(&w.d.y);
  a0 = fmaf(__half2float(t & 1 ? h0.y : h0.x), sum2(s0, s1), a0);
  a1 = fmaf(__half2float(t & 1 ? h1.y : h1.x), sum2(u0, u1), a1);
}

// W warps share the K groups of the CTA's row tile.
template <int QT, int W>
__global__ void __launch_bounds__(W * 32) row_gemv_kernel(const RowGemvParams p) {
  constexpr int TB = tile_bytes(QT), PF = 2;
  extern __shared__ __align__(16) float xs[];           // [kgroups * 4][XB]
  __shared__ float red[W][16], ssq[W];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, g = lane >> 2, t = lane & 3;
  const uint8_t* w = p.w + (size_t)blockIdx.x * p.kgroups * TB;
  LaneTile<QT> pre[PF];
#pragma unroll
  for (int u = 0; u < PF; u++) if (warp + u * W < p.kgroups) pre[u].load(w + (size_t)(warp + u * W) * TB, lane);
  const bool silu = p.epilogue == B200Q_EPI_SILU_MUL;
  const int row = silu ? blockIdx.x * 8 + tid : blockIdx.x * 16 + tid;
  const bool writes = tid < (silu ? 8 : 16) && row < p.n_out;
  pdl_launch_dependents();
  pdl_wait();
  const float bias = writes && p.bias ? __half2float(p.bias[row]) : 0.f, res = writes && p.residual ? p.residual[row] : 0.f;
  float ss = 0.f;
  for (int i = tid * 4; i < p.kgroups * GROUP_ELEMS; i += W * 128) {
    float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
    if (i < p.n_in) {
      v = *reinterpret_cast<const float4*>(p.x + i);
      if (p.norm_w) {
        const uint2 nw = *reinterpret_cast<const uint2*>(p.norm_w + i);
        ss = fmaf(v.x, v.x, fmaf(v.y, v.y, fmaf(v.z, v.z, fmaf(v.w, v.w, ss))));
        const float2 n0 = __half22float2(*reinterpret_cast<const __half2*>(&nw.x)), n1 = __half22float2(*reinterpret_cast<const __half2*>(&nw.y));
        v.x *= n0.x; v.y *= n0.y; v.z *= n1.x; v.w *= n1.y;
      }
    }
    *reinterpret_cast<float4*>(xs + (i >> 5) * XB + (i & 31)) = v;
  }
  __syncthreads();
  float a0 = 0.f, a1 = 0.f;
#pragma unroll
  for (int u = 0; u < PF; u++) if (warp + u * W < p.kgroups) tile_dot<QT>(pre[u], xs + ((warp + u * W) * 4 + t) * XB, t, a0, a1);
#pragma unroll 2
  for (int j = warp + PF * W; j < p.kgroups; j += W) {
    LaneTile<QT> next;
    next.load(w + (size_t)j * TB, lane);
    tile_dot<QT>(next, xs + (j * 4 + t) * XB, t, a0, a1);
  }
  a0 += __shfl_xor_sync(0xffffffffu, a0, 1); a0 += __shfl_xor_sync(0xffffffffu, a0, 2);
  a1 += __shfl_xor_sync(0xffffffffu, a1, 1); a1 += __shfl_xor_sync(0xffffffffu, a1, 2);
  if (t == 0) { red[warp][g] = a0; red[warp][8 + g] = a1; }
  if (p.norm_w) {
    ss = warp_sum(ss);
    if (lane == 0) ssq[warp] = ss;
  }
  __syncthreads();
  if (warp) return;
  float v = 0.f;
  if (lane < 16) {
#pragma unroll
    for (int i = 0; i < W; i++) v += red[i][lane];
  }
  if (p.norm_w) {
    float tot = 0.f;
#pragma unroll
    for (int i = 0; i < W; i++) tot += ssq[i];
    v *= 1.0f / sqrtf(tot / (float)p.n_in + p.eps);
  }
  const float up = __shfl_down_sync(0xffffffffu, v, 8);      // rows 8 .. 15 of an interleaved tile are the `up` rows
  if (!writes) return;
  p.y[row] = silu ? (v / (1.f + expf(-v))) * up : v + bias + res;
}

template <int QT, int W> int launch_row(const RowGemvParams& p, int tiles, cudaStream_t st, bool pdl) {
  const size_t smem = (size_t)p.kgroups * 4 * XB * sizeof(float);
  if (smem > 200 * 1024) return B200Q_ERR_TOO_LARGE;
  static PerDeviceFlag attr_set;
  const int dev = b200q_current_device();
  if (dev < 0) return B200Q_ERR_CUDA;
  if (!attr_set.test(dev)) {
    B200Q_CHECK_CUDA(cudaFuncSetAttribute(row_gemv_kernel<QT, W>, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024));
    attr_set.set(dev);
  }
  B200Q_CHECK_CUDA(launch_k(row_gemv_kernel<QT, W>, dim3(tiles), dim3(W * 32), smem, st, pdl, p));
  return B200Q_OK;
}

}  // namespace

// 4 warps up to 4 K groups, 8 up to 8, else 16: a warp has a tile or two, all of them on their way before the wait.
int b200q_row_gemv_chain(int qtype, const void* w_packed, const float* x, const void* norm_weight, float norm_eps, const void* bias_f16, const float* residual, int epilogue,
                         float* y, int n_out, int n_in, cudaStream_t st, bool pdl) {
  if (!w_packed || !x || !y || n_out <= 0 || n_in <= 0) return B200Q_ERR_BAD_ARG;
  if ((qtype != B200Q_Q4_0 && qtype != B200Q_Q8_0) || (epilogue != B200Q_EPI_LINEAR && epilogue != B200Q_EPI_SILU_MUL)) return B200Q_ERR_BAD_ARG;
  if (epilogue == B200Q_EPI_SILU_MUL && (bias_f16 || residual)) return B200Q_ERR_UNSUPPORTED;
  if (n_in % 32) return B200Q_ERR_BAD_SHAPE;
  if (((uintptr_t)w_packed | (uintptr_t)x) & 15 || (uintptr_t)norm_weight & 7 || ((uintptr_t)y | (uintptr_t)residual) & 3 || (uintptr_t)bias_f16 & 1) return B200Q_ERR_MISALIGNED;
  const RowGemvParams p{(const uint8_t*)w_packed, x, (const __half*)norm_weight, (const __half*)bias_f16, residual, y, n_out, n_in, ceil_div(n_in, GROUP_ELEMS), epilogue, norm_eps};
  const int tiles = ceil_div(n_out, epilogue == B200Q_EPI_SILU_MUL ? 8 : TILE_ROWS);
  if (qtype == B200Q_Q4_0)
    return p.kgroups <= 4 ? launch_row<B200Q_Q4_0, 4>(p, tiles, st, pdl) : p.kgroups <= 8 ? launch_row<B200Q_Q4_0, 8>(p, tiles, st, pdl) : launch_row<B200Q_Q4_0, 16>(p, tiles, st, pdl);
  return p.kgroups <= 4 ? launch_row<B200Q_Q8_0, 4>(p, tiles, st, pdl) : p.kgroups <= 8 ? launch_row<B200Q_Q8_0, 8>(p, tiles, st, pdl) : launch_row<B200Q_Q8_0, 16>(p, tiles, st, pdl);
}

extern "C" int b200q_row_gemv(int qtype, const void* w_packed, const float* x, const void* norm_weight, float norm_eps, const void* bias_f16, const float* residual,
                              int epilogue, float* y, int n_out, int n_in, int flags, void* stream) {
  return b200q_row_gemv_chain(qtype, w_packed, x, norm_weight, norm_eps, bias_f16, residual, epilogue, y, n_out, n_in, (cudaStream_t)stream, flags & B200Q_FLAG_PDL);
}
