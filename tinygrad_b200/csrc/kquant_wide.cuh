// K-quant weights (Q4_K, Q6_K) against activations in full precision: the pieces of the GEMV (gemv.cu) for the block Linears of files that mix
// K-quants.  Weights stay in their file form in memory (4.75 / 6.6 bits each) and become the fp16 values the reference casts every loaded tensor
// to (tinygrad/llm/model.py:376) in registers; an activation is two fp16 numbers, its high part and the remainder times 2^11 (together within
// 2^-23 of the fp32 value).  Products are exact on the tensor cores, sums are fp32.
//
// One tile = 16 rows x 128 columns, eight m16n8k16 fp16 MMAs.  K of an MMA runs over the tile's 4 blocks of 32 (lane t of a quad holds block t: 4
// elements of it per MMA); even columns of B hold the high parts, odd columns the remainders (column pairs 1 .. 3 repeat pair 0, so that all lanes
// of a quad end with the same sums).  A nibble or 6 bits at bit 0 of an fp16 are the subnormal q * 2^-24, at bit 4 q * 2^-20: masks and
// shifts unpack two quants, two conversions and one packed FMA scale them exactly as fp32 would, one conversion rounds the pair to fp16.
// What bounds it is that dequantisation: 64 conversions and 32 packed FMAs on one pipe, 72 masks, shifts and roundings on another per tile, each
// good for an instruction every other cycle.  Gate and up of 14336 x 4096 in Q4_K 26.3 us with running accumulators (2.66 TB/s of packed
// weights; as fp16 these are 235 MB, 36 us at HBM rate; a single cold launch with its events 30.8, and 32.8 with the sums below), down 4096 x 14336 in Q6_K 19.7 us; a step of six 8B-shaped blocks 1005 us on fp16 weights, 510 us here.  Scalar FMAs: 27.0 us.  The mixed-precision FMA on scale * q
// (exact in fp16), which needs no conversions: 30.1 us.
//
// Sums: the tensor core truncates, always towards zero, when it adds to an accumulator, so the high parts' products of two MMAs at a time are added here,
// rounded to nearest.  Error of 4096 x 14336 outputs against 64 bits 1.5e-7, as in fp32 sums on the dense form; with accumulators that run through the MMAs 5.5e-7
// (and 486 us a step).  One MMA at a time is no closer and spills (555 us).
//
// Record of an activation row (kgroups = n_in / 128): uint4 xh[kgroups][4][8], entry w, column c = block (high parts) or 4 + block (remainders):
// {x[4w], x[4w+2]} {x[4w+1], x[4w+3]} and the same of elements 16 + 4w ..; the row is scaled by a power of two that puts its largest value into
// [2^13, 2^14).
#pragma once
#include "qgemv_core.cuh"

namespace {

__host__ __device__ constexpr bool is_wide(int qt) { return qt == B200Q_Q4_K_WIDE || qt == B200Q_Q6_K_WIDE || qt == B200Q_Q4_K_WIDE + B200Q_Q6_K_WIDE; }      // the last: both in one launch

__device__ __forceinline__ uint32_t half2_bits(float a, float b) {
  const __half2 h = __floats2half2_rn(a, b);
  return *reinterpret_cast<const uint32_t*>(&h);
}

// Power of two for a row whose largest magnitude is amax (rows too small to matter count as zero; infinities make the results NaN).
__device__ __forceinline__ void wide_row_scale(float amax, float& up, float& down) {
  const int E = (int)(__float_as_uint(amax) >> 23) - 127;
  const bool live = amax > 1e-30f, huge = !(amax < 1e34f);
  up = huge ? __uint_as_float(0x7FC00000u) : live ? __uint_as_float((uint32_t)(13 - E + 127) << 23) : 0.f;
  down = live && !huge ? __uint_as_float((uint32_t)(E - 13 + 127) << 23) : 0.f;
}
// Elements 8q .. 8q + 7 (q = 0 .. 3) of block b, times `up`.
__device__ __forceinline__ void wide_store_8(const float (&v)[8], int q, int b, float up, unsigned char* xh) {
  const int j = b >> 2, tb = b & 3;
#pragma unroll
  for (int e = 0; e < 2; e++) {
    const int g4 = 2 * q + e, w = g4 & 3, hf = g4 >> 2;
    float hi[4], lo[4];
#pragma unroll
    for (int i = 0; i < 4; i++) {
      const float s = v[4 * e + i] * up;
      hi[i] = __half2float(__float2half_rn(s));
      lo[i] = (s - hi[i]) * 2048.f;
    }
    unsigned char* at = xh + (((size_t)j * 4 + w) * 8 + tb) * 16 + hf * 8;
    *reinterpret_cast<uint2*>(at) = make_uint2(half2_bits(hi[0], hi[2]), half2_bits(hi[1], hi[3]));
    *reinterpret_cast<uint2*>(at + 64) = make_uint2(half2_bits(lo[0], lo[2]), half2_bits(lo[1], lo[3]));
  }
}

// c += A (16 x 16) B (16 x 8)
__device__ __forceinline__ void hmma(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
  asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
               : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3]) : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
// Two quants (as fp16 subnormals) -> two weights: q * a + b in fp32 (one packed FMA), rounded to fp16.
struct PairFma {
  unsigned long long a, b;
  __device__ __forceinline__ PairFma(float av, float bv) {
    asm("mov.b64 %0, {%1, %1};" : "=l"(a) : "f"(av));
    asm("mov.b64 %0, {%1, %1};" : "=l"(b) : "f"(bv));
  }
  __device__ __forceinline__ uint32_t operator()(uint32_t q) const {
    uint32_t r;
    asm("{.reg .b16 l, h;\n.reg .f32 x, y;\n.reg .b64 v;\nmov.b32 {l, h}, %1;\ncvt.f32.f16 x, l;\ncvt.f32.f16 y, h;\nmov.b64 v, {x, y};\n"
        "fma.rn.f32x2 v, v, %2, %3;\nmov.b64 {x, y}, v;\ncvt.rn.f16x2.f32 %0, y, x;}" : "=r"(r) : "r"(q), "l"(a), "l"(b));
    return r;
  }
};
constexpr float SUB0 = 16777216.f, SUB4 = 1048576.f;      // 2^24, 2^20: what quants at bit 0 / bit 4 of an fp16 lack

// One Q4_K tile, 1216 bytes: uint4 L[2][32] quants (lane (g, t) of half h: row 8h + g, block t; byte i = element i | element i + 16 << 4),
// uint8 SM[16][4][2] {scale, minimum} of each block, half2 D[16] {d, dmin}.  Weight = d * scale * q - dmin * minimum (tinygrad/llm/gguf.py:57-67).
// xb: the lane's column and block of the group's xh entries, 8 entries apart.
__device__ __forceinline__ void tile_mac_q4k(const uint8_t* tile, int lane, const uint4* xb, float (&c)[4]) {
  const uint4* lp = reinterpret_cast<const uint4*>(tile);
  const uint4 r0 = lp[lane], r1 = lp[32 + lane];      // rows g and g + 8
  const int g = lane >> 2;
  const uint32_t s0 = *reinterpret_cast<const uint16_t*>(tile + 1024 + lane * 2), s1 = *reinterpret_cast<const uint16_t*>(tile + 1024 + 64 + lane * 2);
  const float2 d0 = __half22float2(reinterpret_cast<const __half2*>(tile + 1152)[g]), d1 = __half22float2(reinterpret_cast<const __half2*>(tile + 1152)[g + 8]);
  const float b0 = -d0.y * (float)(s0 >> 8), b1 = -d1.y * (float)(s1 >> 8);
  constexpr uint32_t LO = 0x000F000Fu, HI = 0x00F000F0u;
  const uint32_t w0[4] = {r0.x, r0.y, r0.z, r0.w}, w1[4] = {r1.x, r1.y, r1.z, r1.w};
  const float a0 = d0.x * (float)(s0 & 0xFF), a1 = d1.x * (float)(s1 & 0xFF);
  const PairFma lo0(a0 * SUB0, b0), lo1(a1 * SUB0, b1), hi0(a0 * SUB4, b0), hi1(a1 * SUB4, b1);
#pragma unroll
  for (int w = 0; w < 4; w++) {
    const uint4 x = xb[w * 8];
    const uint32_t u0 = w0[w] >> 8, u1 = w1[w] >> 8;
    float p[4] = {0.f, c[1], 0.f, c[3]};
    hmma(p, lo0(w0[w] & LO), lo1(w1[w] & LO), lo0(u0 & LO), lo1(u1 & LO), x.x, x.y);
    hmma(p, hi0(w0[w] & HI), hi1(w1[w] & HI), hi0(u0 & HI), hi1(u1 & HI), x.z, x.w);
    c[0] += p[0]; c[1] = p[1]; c[2] += p[2]; c[3] = p[3];
  }
}

// One Q6_K tile in the layout of tile_mac_q6k: weight = d * scale * (q - 32).
__device__ __forceinline__ void tile_mac_q6k_wide(const uint8_t* tile, int lane, const uint4* xb, float (&c)[4]) {
  const uint4* lp = reinterpret_cast<const uint4*>(tile);
  const uint2* hp = reinterpret_cast<const uint2*>(tile + 1024);
  const uint4 r0 = lp[lane], r1 = lp[32 + lane];      // rows g and g + 8
  const uint2 h0 = hp[lane], h1 = hp[32 + lane];
  const int g = lane >> 2;
  const char2 s0 = *reinterpret_cast<const char2*>(tile + 1536 + lane * 2), s1 = *reinterpret_cast<const char2*>(tile + 1536 + 64 + lane * 2);
  const __half* dp = reinterpret_cast<const __half*>(tile + 1664);
  const float d0 = __half2float(dp[g]), d1 = __half2float(dp[g + 8]);
  const float a0 = d0 * (float)s0.x, e0 = d0 * (float)s0.y, a1 = d1 * (float)s1.x, e1 = d1 * (float)s1.y;
  const PairFma lo0(a0 * SUB0, -32.f * a0), lo1(a1 * SUB0, -32.f * a1), hi0(e0 * SUB4, -32.f * e0), hi1(e1 * SUB4, -32.f * e1);
  constexpr uint32_t LO = 0x000F000Fu, HI = 0x00F000F0u, LO2 = 0x00300030u, HI2 = 0x03000300u;
  const uint32_t w0[4] = {r0.x, r0.y, r0.z, r0.w}, w1[4] = {r1.x, r1.y, r1.z, r1.w};
  // the bit pair of element 4w + k sits at bits 2w of byte k: to bits 4 (first half of a block) or 8 (second) of each fp16
  auto sh = [](uint32_t v, int n) { return n >= 0 ? v << n : v >> -n; };
#pragma unroll
  for (int w = 0; w < 4; w++) {
    const uint4 x = xb[w * 8];
    const uint32_t u0 = w0[w] >> 8, u1 = w1[w] >> 8;
    float p[4] = {0.f, c[1], 0.f, c[3]};
    hmma(p, lo0((w0[w] & LO) | (sh(h0.x, 4 - 2 * w) & LO2)), lo1((w1[w] & LO) | (sh(h1.x, 4 - 2 * w) & LO2)),
         lo0((u0 & LO) | (sh(h0.x, -4 - 2 * w) & LO2)), lo1((u1 & LO) | (sh(h1.x, -4 - 2 * w) & LO2)), x.x, x.y);
    hmma(p, hi0((w0[w] & HI) | (sh(h0.y, 8 - 2 * w) & HI2)), hi1((w1[w] & HI) | (sh(h1.y, 8 - 2 * w) & HI2)),
         hi0((u0 & HI) | (sh(h0.y, -2 * w) & HI2)), hi1((u1 & HI) | (sh(h1.y, -2 * w) & HI2)), x.z, x.w);
    c[0] += p[0]; c[1] = p[1]; c[2] += p[2]; c[3] = p[3];
  }
}

}  // namespace
