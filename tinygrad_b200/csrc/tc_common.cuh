// Pieces shared by the tcgen05 dequant GEMMs: operand descriptors, bounded mbarrier waits and the unpacking of Q4_0 / Q8_0 blocks into
// fp16 operand chunks.
#pragma once
#include "common.cuh"

namespace {

constexpr int SPIN = 1 << 22;

__device__ int g_tc_status = 0;                         // one per translation unit: 1 = a bounded wait ran out

__device__ __forceinline__ uint32_t s32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

// shared-memory matrix descriptor, K-major, no swizzle: core matrix = 8 rows x 16 bytes, stored as 128 contiguous bytes;
// LBO = byte distance between core matrices adjacent in K, SBO = between core matrices adjacent in M/N.
__device__ __forceinline__ uint64_t make_desc(uint32_t saddr, uint32_t lbo, uint32_t sbo) {
  uint64_t d = 0;
  d |= (uint64_t)((saddr >> 4) & 0x3FFF);
  d |= (uint64_t)((lbo >> 4) & 0x3FFF) << 16;
  d |= (uint64_t)((sbo >> 4) & 0x3FFF) << 32;
  d |= (uint64_t)1 << 46;                       // descriptor version of this architecture
  return d;                                     // base offset 0, layout type 0 (no swizzle)
}
// instruction descriptor, kind::f16: fp16 x fp16 -> fp32, both operands K-major
__device__ __forceinline__ uint32_t make_idesc(int m, int n) {
  return (1u << 4) | (0u << 7) | (0u << 10) | ((uint32_t)(n >> 3) << 17) | ((uint32_t)(m >> 4) << 24);
}

__device__ __forceinline__ bool wait_bar(uint32_t bar, uint32_t parity) {
  for (int i = 0; i < SPIN; i++) {
    uint32_t ok;
    asm volatile("{\n.reg .pred p;\nmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\nselp.u32 %0, 1, 0, p;\n}" : "=r"(ok) : "r"(bar), "r"(parity) : "memory");
    if (ok) return true;
  }
  atomicExch(&g_tc_status, 1);
  return false;
}

// element (r, k) of an R-row tile: core (r/8, k/8) at (k/8) * (R*16) + (r/8) * 128, inside the core (r%8)*16 + (k%8)*2 bytes
__device__ __forceinline__ uint32_t tile_off(int r, int k, int rows) { return (k >> 3) * (rows * 16) + (r >> 3) * 128 + (r & 7) * 16 + (k & 7) * 2; }

__device__ __forceinline__ uint32_t lop3_and_or(uint32_t a, uint32_t b, uint32_t c) { uint32_t d; asm("lop3.b32 %0, %1, %2, %3, 0xEA;" : "=r"(d) : "r"(a), "r"(b), "r"(c)); return d; }
__device__ __forceinline__ uint32_t h2sub(uint32_t a, uint32_t b) { uint32_t d; asm("sub.f16x2 %0, %1, %2;" : "=r"(d) : "r"(a), "r"(b)); return d; }
__device__ __forceinline__ uint32_t h2mul(uint32_t a, uint32_t b) { uint32_t d; asm("mul.f16x2 %0, %1, %2;" : "=r"(d) : "r"(a), "r"(b)); return d; }
__device__ __forceinline__ uint32_t h2fma(uint32_t a, uint32_t b, uint32_t c) { uint32_t d; asm("fma.rn.f16x2 %0, %1, %2, %3;" : "=r"(d) : "r"(a), "r"(b), "r"(c)); return d; }
__device__ __forceinline__ uint32_t prmt(uint32_t a, uint32_t b, uint32_t sel) { uint32_t d; asm("prmt.b32 %0, %1, %2, %3;" : "=r"(d) : "r"(a), "r"(b), "r"(sel)); return d; }

__device__ __forceinline__ uint32_t h2fma_neg(uint32_t a, uint32_t b, uint32_t c) {      // a * b - c (the sign costs nothing inside the instruction)
  uint32_t d;
  asm("{\n.reg .b32 n;\nneg.f16x2 n, %3;\nfma.rn.f16x2 %0, %1, %2, n;\n}" : "=r"(d) : "r"(a), "r"(b), "r"(c));
  return d;
}

// q * d for four pairs: the fp16 product (hi, = the reference's materialised fp16 weight) and its exact remainder
// lo = q * d - hi (one fused multiply-add: the remainder has at most 8 significant bits, so it is exact).  hi + lo is the
// fp32 value the reference's fused kernels use when the activations are fp32 (tinygrad/codegen/late/coalesce.py:100).
__device__ __forceinline__ uint4 hi_lo(const uint32_t (&r)[4], uint32_t d2, uint4& lo) {
  const uint4 hi = make_uint4(h2mul(r[0], d2), h2mul(r[1], d2), h2mul(r[2], d2), h2mul(r[3], d2));
  lo = make_uint4(h2fma_neg(r[0], d2, hi.x), h2fma_neg(r[1], d2, hi.y), h2fma_neg(r[2], d2, hi.z), h2fma_neg(r[3], d2, hi.w));
  return hi;
}
// 8 nibbles of two words (bytes 0..7 of a 16-byte half) -> one core row of 8 fp16 weights, low (HI = false) or high nibbles
template <bool HI>
__device__ __forceinline__ uint4 q4_core(uint32_t wa, uint32_t wb, uint32_t d2, uint4& lo) {
  const uint32_t MAGIC = 0x64006400u;
  uint32_t r[4];
  const uint32_t w[2] = {wa, wb};
#pragma unroll
  for (int i = 0; i < 2; i++) {
    const uint32_t v = w[i] >> 8;
    if (!HI) {   // (1024 + n) - 1032 = n - 8
      r[2 * i] = h2sub(lop3_and_or(w[i], 0x000F000Fu, MAGIC), 0x64086408u);
      r[2 * i + 1] = h2sub(lop3_and_or(v, 0x000F000Fu, MAGIC), 0x64086408u);
    } else {     // (1024 + 16 n) / 16 - 72 = n - 8
      r[2 * i] = h2fma(lop3_and_or(w[i], 0x00F000F0u, MAGIC), 0x2C002C00u, 0xD480D480u);
      r[2 * i + 1] = h2fma(lop3_and_or(v, 0x00F000F0u, MAGIC), 0x2C002C00u, 0xD480D480u);
    }
  }
  return hi_lo(r, d2, lo);
}
// 8 int8 of two words -> one core row of 8 fp16 weights
__device__ __forceinline__ uint4 q8_core(uint32_t wa, uint32_t wb, uint32_t d2, uint4& lo) {
  const uint32_t HIB = 0x64646464u, SUB = 0x64806480u;     // 0x64bb = 1024 + (b ^ 0x80) = 1152 + b
  const uint32_t xa = wa ^ 0x80808080u, xb = wb ^ 0x80808080u;
  const uint32_t r[4] = {h2sub(prmt(xa, HIB, 0x4240u), SUB), h2sub(prmt(xa, HIB, 0x4341u), SUB), h2sub(prmt(xb, HIB, 0x4240u), SUB),
                         h2sub(prmt(xb, HIB, 0x4341u), SUB)};
  return hi_lo(r, d2, lo);
}
// the 8 nibbles of a word (4 bytes of a block: low nibbles = elements i .. i + 3, high nibbles = elements i + 16 ..) as fp16 pairs of q - 8:
// a nibble in bits 0..3 under the exponent of 1024 reads 1024 + q, in bits 4..7 under that of 64 it reads 64 + q.  One shift, no multiply.
__device__ __forceinline__ void q4_word(uint32_t w, uint32_t (&v)[4]) {      // v: {e0,e2}, {e1,e3}, {e16,e18}, {e17,e19}
  const uint32_t u = w >> 8;
  v[0] = h2sub(lop3_and_or(w, 0x000F000Fu, 0x64006400u), 0x64086408u);
  v[1] = h2sub(lop3_and_or(u, 0x000F000Fu, 0x64006400u), 0x64086408u);
  v[2] = h2sub(lop3_and_or(w, 0x00F000F0u, 0x54005400u), 0x54805480u);
  v[3] = h2sub(lop3_and_or(u, 0x00F000F0u, 0x54005400u), 0x54805480u);
}

// 8 fp32 values -> a chunk of 8 fp16 high parts and one of the remainders' fp16 roundings, in the unpack's element order
__device__ __forceinline__ void split_chunk(const float (&f)[8], uint4& hi, uint4& lo) {
  const __half2 o[4] = {__floats2half2_rn(f[0], f[2]), __floats2half2_rn(f[1], f[3]), __floats2half2_rn(f[4], f[6]), __floats2half2_rn(f[5], f[7])};
  const float2 h0 = __half22float2(o[0]), h1 = __half22float2(o[1]), h2 = __half22float2(o[2]), h3 = __half22float2(o[3]);
  const __half2 l[4] = {__floats2half2_rn(f[0] - h0.x, f[2] - h0.y), __floats2half2_rn(f[1] - h1.x, f[3] - h1.y),
                        __floats2half2_rn(f[4] - h2.x, f[6] - h2.y), __floats2half2_rn(f[5] - h3.x, f[7] - h3.y)};
  hi = *reinterpret_cast<const uint4*>(o);
  lo = *reinterpret_cast<const uint4*>(l);
}

}  // namespace
