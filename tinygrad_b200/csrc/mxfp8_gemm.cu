// Grouped (per-expert) MXFP8 GEMM on the 5th-generation tensor cores:
//   C[M, N] (bf16) = A_q[M, K] (e4m3) x B_q[e(row)][N, K]^T (e4m3), one E8M0 scale per 32 along K on both operands, fp32 accumulation.
// Rows of A are grouped by expert: group e = rows off[e] .. off[e+1], every group a multiple of 256 rows.
// Semantics: extra/gemm/moe_gemm.py:112-134 over the kernel contract of extra/thunder/amd/grouped_mxfp8_gemm.cpp:32-158
// (the reference computation it is tested against: dequantised operands matmul, test/backend/test_asm_gemm.py:289-292,306).
//
// Persistent, warp-specialised kernel, one CTA per SM, 128 x 256 output tiles (128 x 128 or x 64 where those are too few for the SMs: tile_columns), tiles of the used
// rows (off[E]) dealt round-robin:
//   warps 4-7  loaders: one thread brings the A (128 x 128 B) and B (256 x 128 B) tiles of a K step into a ring of 3 to 5 stages by tensor-map copies (K-major, 128-byte
//              swizzle: 16-byte chunk c of row r sits at chunk c ^ (r & 7)), all of them the step's E8M0 scale words by cp.async (one 32-bit
//              word = 4 K blocks per row, stored as 32 x 16 B chunks: row r -> chunk r % 32, word r / 32); the copies' bytes and each thread's
//              words arrive on the stage's "full" mbarrier when they land (no scale words where all of them are one: UNIT);
//   warp 8     one thread moves the scale chunks to tensor memory with tcgen05.cp 32x128b.warpx4 (row r -> lane r % 32 of every
//              32-lane sub-partition, column r / 32: the layout the MMA reads), issues tcgen05.mma kind::mxf8f6f4.block_scale
//              (scale_vec::1X, 128 x 256 x 32 per instruction, the tensor core applies both block scales), four per K step, and
//              commits each step to the stage's "empty" mbarrier;
//   warps 0-3, 9-20  epilogue: tcgen05.ld the fp32 accumulator (256 tensor-memory columns; four warps per 32-lane sub-partition,
//              64 columns each) into registers, release the accumulator, then one of four endings (OUT_BF16 ..).
// Loaders run ahead across tile boundaries; the accumulator (one buffer at every tile width: two of 256 columns and the scale columns do not fit the 512 of
// tensor memory, and with narrower tiles a CTA has one or few) is handed back after one tensor-memory round trip, the epilogue's arithmetic and stores overlap the next tile's MMAs.
// Every mbarrier wait is bounded; a wait that runs out raises a status word and makes every role leave.
#include "common.cuh"
#include "mxq.cuh"
#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <algorithm>

namespace {

constexpr int BM = 128, BN_MAX = 256, BK = 128, FEW_ROWS = 32;
constexpr int EPI_WARPS = 4, LOAD_WARPS = 4, EPI_Q = 4;      // epilogue: warps 0-3 and 9-20, EPI_Q warps per 32-lane sub-partition (64 columns each)
constexpr int THREADS = (EPI_Q * EPI_WARPS + LOAD_WARPS + 1) * 32;
constexpr int EPI_STAGE_BYTES = 16 * 4096;                                              // staging rows of the epilogues that store by tensor-map copies (bf16, FP8 linear): 4 KB per warp
constexpr int TMEM_COLS = 512;            // 256 accumulator columns + scale columns, rounded up to a power of two
// The tile's columns: a ring stage holds 128 rows of A, BN of B and the scale chunks (A 512 B, B 2 x 512 B), a multiple of 1024 bytes: 50, 34 or 26 KB
template <int BN> struct Geo {
  static constexpr int STAGES = BN == 256 ? 3 : BN == 128 ? 4 : 5;
  static constexpr int A_BYTES = BM * BK, B_BYTES = BN * BK, SF_BYTES = 2048, STAGE_BYTES = A_BYTES + B_BYTES + SF_BYTES;
  static constexpr int SMEM_BYTES = STAGES * STAGE_BYTES + 1024 + EPI_STAGE_BYTES;        // + room to align the ring to 1024 B
  static_assert(SMEM_BYTES + 9 * 1024 <= 227 * 1024, "with the tables of groups");
  static constexpr int SFA_COL = 256, SFB_COL = 256 + 4 * STAGES;   // tensor-memory columns, per stage 4 (A: 128 rows) and 8 (B: 256 rows)
};
constexpr int MAX_EXPERTS = 1024;
constexpr int SPIN = 1 << 22;

__device__ int g_mx_status = 0;

__device__ __forceinline__ uint32_t s32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void cp4(uint32_t s, const void* g) { asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(s), "l"(g) : "memory"); }
__device__ __forceinline__ uint64_t desc_plain(uint32_t saddr, uint32_t lbo, uint32_t sbo) {
  uint64_t d = 0;
  d |= (uint64_t)((saddr >> 4) & 0x3FFF);
  d |= (uint64_t)((lbo >> 4) & 0x3FFF) << 16;      // core matrices adjacent in K
  d |= (uint64_t)((sbo >> 4) & 0x3FFF) << 32;      // core matrices adjacent in M / N
  d |= (uint64_t)1 << 46;
  return d;
}
// K-major, 128-byte swizzle: 8-row groups 1024 B apart; a K offset inside the 128-byte row is added to the start address
__device__ __forceinline__ uint64_t desc_sw128(uint32_t saddr) {
  uint64_t d = 0;
  d |= (uint64_t)((saddr >> 4) & 0x3FFF);
  d |= (uint64_t)1 << 16;
  d |= (uint64_t)(1024 >> 4) << 32;
  d |= (uint64_t)1 << 46;
  d |= (uint64_t)2 << 61;
  return d;
}
__device__ __forceinline__ bool wait_bar(uint32_t bar, uint32_t parity, volatile int* abort_flag) {
#pragma unroll 1
  for (int i = 0; i < SPIN; i++) {
    uint32_t ok;
    asm volatile("{\n.reg .pred p;\nmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\nselp.u32 %0, 1, 0, p;\n}" : "=r"(ok) : "r"(bar), "r"(parity) : "memory");
    if (ok) return true;
    if ((i & 255) == 255 && *abort_flag) return false;
  }
  *abort_flag = 1;
  atomicExch(&g_mx_status, 1);
  return false;
}
__device__ __forceinline__ void arrive(uint32_t bar) { asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory"); }

// 32 consecutive accumulator columns of this thread's row (tensor-memory lane) -> registers; the caller waits (tcgen05.wait::ld)
__device__ __forceinline__ void tmem_ld32(uint32_t ta, uint32_t (&v)[32]) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];"
               : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]), "=r"(v[8]), "=r"(v[9]), "=r"(v[10]),
                 "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15]), "=r"(v[16]), "=r"(v[17]), "=r"(v[18]), "=r"(v[19]), "=r"(v[20]),
                 "=r"(v[21]), "=r"(v[22]), "=r"(v[23]), "=r"(v[24]), "=r"(v[25]), "=r"(v[26]), "=r"(v[27]), "=r"(v[28]), "=r"(v[29]), "=r"(v[30]),
                 "=r"(v[31])
               : "r"(ta));
}
// one MX block of the activation: gate / up accumulators of 32 columns -> silu(gate) * up -> E4M3 codes + block exponent at [row, col..col+31]
__device__ __forceinline__ void swiglu_quant_store(const uint32_t (&vg)[32], const uint32_t (&vu)[32], uint8_t* act_q, uint8_t* act_e8, size_t row, int f,
                                                   int col) {
  float v[32];
  float amax = 0.f;
#pragma unroll
  for (int j = 0; j < 32; j++) {
    const float g = __bfloat162float(__float2bfloat16_rn(__uint_as_float(vg[j]))), u = __bfloat162float(__float2bfloat16_rn(__uint_as_float(vu[j])));
    v[j] = __bfloat162float(__float2bfloat16_rn((g / (1.f + expf(-g))) * u));
    amax = fmaxf(amax, fabsf(v[j]));
  }
  const uint8_t e = mx_scale_exponent(amax);
  uint2 pk[4];
#pragma unroll
  for (int q = 0; q < 4; q++) {
    const float v8[8] = {v[8 * q], v[8 * q + 1], v[8 * q + 2], v[8 * q + 3], v[8 * q + 4], v[8 * q + 5], v[8 * q + 6], v[8 * q + 7]};
    pk[q] = mx_quant8(v8, e);
  }
  uint4* dst = reinterpret_cast<uint4*>(act_q + row * f + col);
  dst[0] = make_uint4(pk[0].x, pk[0].y, pk[1].x, pk[1].y);
  dst[1] = make_uint4(pk[2].x, pk[2].y, pk[3].x, pk[3].y);
  act_e8[row * (f >> 5) + (col >> 5)] = e;
}

// The same for the first `rows` rows of a narrow tile with few: the warp's accumulators (a row per lane, 32 gate and 32 up columns) change places in shared memory, then a
// row's block is a value per lane.  With a row per lane and everything unrolled, one token's tiles were mostly the time to fetch 3000 instructions.
__device__ __forceinline__ void swiglu_quant_few(const uint32_t (&vg)[32], const uint32_t (&vu)[32], float* s, uint8_t* act_q, uint8_t* act_e8, size_t row0, int rows, int f, int col) {
  const int lane = threadIdx.x & 31;
  constexpr int STRIDE = 65;
  if (lane < rows) {
#pragma unroll
    for (int j = 0; j < 32; j++) { s[lane * STRIDE + j] = __uint_as_float(vg[j]); s[lane * STRIDE + 32 + j] = __uint_as_float(vu[j]); }
  }
  __syncwarp();
#pragma unroll 1
  for (int r = 0; r < rows; r++) {
    const float g = __bfloat162float(__float2bfloat16_rn(s[r * STRIDE + lane])), u = __bfloat162float(__float2bfloat16_rn(s[r * STRIDE + 32 + lane]));
    const float v = __bfloat162float(__float2bfloat16_rn((g / (1.f + expf(-g))) * u));
    const uint8_t e = mx_scale_exponent(warp_max(fabsf(v)));
    act_q[(row0 + r) * f + col + lane] = __nv_cvt_float_to_fp8(fminf(fmaxf(v * mx_inv_scale(e), -448.f), 448.f), __NV_SATFINITE, __NV_E4M3);
    if (lane == 0) act_e8[(row0 + r) * (f >> 5) + (col >> 5)] = e;
  }
  __syncwarp();
}

// fp32 results with the per-tensor FP8 linear's last steps: y = acc * *fw * *fx + bias in y's type, for the first `rows` rows (fw NULL: plain sums)
struct ScaledOut { const float *fw, *fx, *bias; int rows, y_f16; };

// What becomes of the sums: bf16 rows, SwiGLU of gate and up requantised, the FP8 linear's results, fp32 sums.  One kernel each: the registers of one epilogue are not
// another's, and an expert layer of few rows does not fetch the instructions of all four.
enum { OUT_BF16, OUT_SWIGLU, OUT_SCALED, OUT_F32 };
// UNIT: every block scale is one (the FP8 linear): they are put into tensor memory once, not brought in with every K step.
// a_rows (BN 64): rows of A that a tile's copies bring, 128 or FEW_ROWS (then every group has at most that many, and the other lanes' results are dropped).
template <int OUT, int BN>
__global__ void __launch_bounds__(THREADS, 1) grouped_mxfp8_tc_kernel(const uint8_t* __restrict__ a_q, const uint8_t* __restrict__ a_e8,
                                                                      const uint8_t* __restrict__ b_q, const uint8_t* __restrict__ b_e8,
                                                                      const int32_t* __restrict__ off, int n_experts, int m_total, int n, int k,
                                                                      __nv_bfloat16* __restrict__ c, uint8_t* __restrict__ act_q,
                                                                      uint8_t* __restrict__ act_e8, const __grid_constant__ CUtensorMap tm_a,
                                                                      const __grid_constant__ CUtensorMap tm_b, const __grid_constant__ CUtensorMap tm_c,
                                                                      const ScaledOut so, const int32_t* __restrict__ ends, int a_rows) {
  using G = Geo<BN>;
  constexpr int STAGES = G::STAGES, A_BYTES = G::A_BYTES, B_BYTES = G::B_BYTES, STAGE_BYTES = G::STAGE_BYTES, SFA_COL = G::SFA_COL, SFB_COL = G::SFB_COL;
  constexpr bool UNIT = OUT == OUT_SCALED, PAIRED = OUT == OUT_SWIGLU && BN < 256;      // PAIRED: half the tile's rows of B are gate rows, the other half lies 128 rows on
  extern __shared__ unsigned char sm_raw[];
  __shared__ __align__(8) uint64_t bar_full[STAGES], bar_empty[STAGES], bar_acc_full, bar_acc_empty, bar_drain;
  __shared__ uint32_t tmem_base;
  __shared__ int s_abort;
  __shared__ int s_off[MAX_EXPERTS], s_tile[MAX_EXPERTS + 1];       // first row of each group, row tiles before it
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  if (tid == 0) {
    for (int s = 0; s < STAGES; s++) {
      asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(s32(&bar_full[s])), "r"(UNIT ? 1 : LOAD_WARPS * 32 + 1));
      asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(s32(&bar_empty[s])));
    }
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(s32(&bar_acc_full)));
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(s32(&bar_acc_empty)), "r"(EPI_Q * EPI_WARPS));
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(s32(&bar_drain)));
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    s_abort = 0;
  }
  if (tid == EPI_WARPS * 32) {
    asm volatile("prefetch.tensormap [%0];" ::"l"(&tm_a) : "memory");
    asm volatile("prefetch.tensormap [%0];" ::"l"(&tm_b) : "memory");
  }
  if (warp == EPI_WARPS + LOAD_WARPS) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(s32(&tmem_base)), "r"(TMEM_COLS) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  pdl_wait();                                       // everything above runs under the previous kernel's tail
  // row tiles of the rows each group has (`ends`: without its padding); everything else of the padded layout is left alone
  if (warp == 0) {
    int carry = 0;
#pragma unroll 1
    for (int e0 = 0; e0 < n_experts; e0 += 32) {
      const int e = e0 + lane;
      int lo = 0, tiles = 0;
      if (e < n_experts) {
        lo = min(max(off[e], 0), m_total);
        int hi = min(max(ends ? ends[e] : off[e + 1], lo), m_total);
        if (OUT == OUT_SCALED) hi = min(hi, max(so.rows, lo));
        tiles = min((hi - lo + BM - 1) / BM, (m_total - lo) / BM);
      }
      int incl = tiles;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) { const int v = __shfl_up_sync(0xffffffffu, incl, o); if (lane >= o) incl += v; }
      if (e < n_experts) { s_off[e] = lo; s_tile[e] = carry + incl - tiles; }
      carry += __shfl_sync(0xffffffffu, incl, 31);
    }
    if (lane == 0) s_tile[n_experts] = carry;
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  pdl_launch_dependents();
  const uint32_t taddr = tmem_base;
  if constexpr (UNIT) {
    if (warp < 4) {      // E8M0 127 = 2^0 in all twelve columns, a warp per sub-partition
      const uint32_t one = 0x7F7F7F7Fu, at = taddr + ((uint32_t)(warp * 32) << 16);
      asm volatile("tcgen05.st.sync.aligned.32x32b.x4.b32 [%0], {%1, %1, %1, %1};" ::"r"(at + SFA_COL), "r"(one) : "memory");
      asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1, %1, %1, %1, %1, %1, %1, %1};" ::"r"(at + SFB_COL), "r"(one) : "memory");
      asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
      asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    }
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  }
  volatile int* abort_flag = &s_abort;
  const int kb_total = k >> 5, ktiles = k / BK;
  const int tiles_n = n / BN, n_tiles = s_tile[n_experts] * tiles_n;
  auto group_of = [&](int mt) {                     // the group whose row tile `mt` is
    int lo = 0, hi = n_experts - 1;
    while (lo < hi) { const int mid = (lo + hi) >> 1; if (s_tile[mid + 1] <= mt) lo = mid + 1; else hi = mid; }
    return lo;
  };
  const uint32_t ring = (s32(sm_raw) + 1023u) & ~1023u;

  if (warp >= EPI_WARPS && warp < EPI_WARPS + LOAD_WARPS) {
    // ---------------------------------------------------------------- loaders
    const int lt = tid - EPI_WARPS * 32;            // 0..127
    const uint32_t sf_off = (uint32_t)((lt & 31) * 16 + (lt >> 5) * 4);      // scale word of row lt (A), rows lt and lt + 128 (B)
    int b_row0 = 0, a_row0 = 0;      // first rows of the tile's operands: B inside [n_experts * n, k], A inside [m_total, k]
    auto tile_ptrs = [&](int t, const uint8_t*& ae, const uint8_t*& be) {
      const int mt = t / tiles_n, n0 = (t % tiles_n) * BN, lo = group_of(mt), m0 = s_off[lo] + (mt - s_tile[lo]) * BM;
      b_row0 = lo * n + (PAIRED ? (n0 >> 8) * 256 + ((n0 >> 1) & 127) : n0); a_row0 = m0;
      ae = a_e8 + (size_t)(m0 + lt) * kb_total;
      be = b_e8 + ((size_t)b_row0 + (PAIRED && lt >= BN / 2 ? 128 - BN / 2 : 0) + lt) * kb_total;
    };
    const uint32_t step_bytes = BN == 64 ? (uint32_t)a_rows * BK + B_BYTES : A_BYTES + B_BYTES;
    uint32_t g = 0;
    bool ok = true;
#pragma unroll 1
    for (int t = blockIdx.x; t < n_tiles && ok; t += gridDim.x) {
      const uint8_t *ae, *be;
      tile_ptrs(t, ae, be);
#pragma unroll 1
      for (int kt = 0; kt < ktiles; kt++, g++) {
        const uint32_t slot = g % STAGES;
        if (g >= STAGES && !wait_bar(s32(&bar_empty[slot]), ((g / STAGES) - 1) & 1, abort_flag)) { ok = false; break; }
        const uint32_t sA = ring + slot * STAGE_BYTES, sB = sA + A_BYTES, sF = sB + B_BYTES;
        __syncwarp();
        if (warp == EPI_WARPS && elect_one()) {
          // the 128-byte-swizzle tiled copy writes exactly the layout above (chunk c of row r at c ^ (r & 7)); no multicast
          const uint32_t fb = s32(&bar_full[slot]);
          asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(fb), "r"(step_bytes) : "memory");
          asm volatile("cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];"
                       ::"r"(sA), "l"(&tm_a), "r"(kt * BK), "r"(a_row0), "r"(fb) : "memory");
          asm volatile("cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];"
                       ::"r"(sB), "l"(&tm_b), "r"(kt * BK), "r"(b_row0), "r"(fb) : "memory");
          if (PAIRED)
            asm volatile("cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];"
                         ::"r"(sB + B_BYTES / 2), "l"(&tm_b), "r"(kt * BK), "r"(b_row0 + 128), "r"(fb) : "memory");
        }
        if constexpr (!UNIT) {
          cp4(sF + sf_off, ae + kt * 4);
          if (BN >= 128 || lt < BN) cp4(sF + 512 + sf_off, be + kt * 4);
          if (BN == 256) cp4(sF + 1024 + sf_off, be + (size_t)128 * kb_total + kt * 4);
          asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];" ::"r"(s32(&bar_full[slot])) : "memory");
        }
      }
    }
    asm volatile("cp.async.wait_all;" ::: "memory");
    // nothing of this thread's tensor-map copies may still be landing when the CTA leaves (they are all consumed unless a wait ran out)
    if (lt == 0)
      for (uint32_t j = g > STAGES ? g - STAGES : 0; j < g; j++) {
        const uint32_t fb = s32(&bar_full[j % STAGES]), par = (j / STAGES) & 1;
#pragma unroll 1
        for (int i = 0; i < SPIN; i++) {
          uint32_t done;
          asm volatile("{\n.reg .pred p;\nmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\nselp.u32 %0, 1, 0, p;\n}" : "=r"(done) : "r"(fb), "r"(par) : "memory");
          if (done) break;
        }
      }
  } else if (warp == EPI_WARPS + LOAD_WARPS) {
    // ---------------------------------------------------------------- MMA issue (one thread)
    if (elect_one()) {
      uint32_t g = 0, tile_i = 0;
      bool ok = true;
#pragma unroll 1
      for (int t = blockIdx.x; t < n_tiles && ok; t += gridDim.x, tile_i++) {
        if (tile_i > 0 && !wait_bar(s32(&bar_acc_empty), (tile_i - 1) & 1, abort_flag)) { ok = false; break; }
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
#pragma unroll 1
        for (int kt = 0; kt < ktiles; kt++, g++) {
          const uint32_t slot = g % STAGES;
          if (!wait_bar(s32(&bar_full[slot]), (g / STAGES) & 1, abort_flag)) { ok = false; break; }
          asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
          asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
          const uint32_t sA = ring + slot * STAGE_BYTES, sB = sA + A_BYTES, sF = sB + B_BYTES;
          // scale chunks -> tensor memory (32 lanes x 16 B, replicated into the four sub-partitions); ordered before the MMAs below
          if constexpr (!UNIT) {
            asm volatile("tcgen05.cp.cta_group::1.32x128b.warpx4 [%0], %1;" ::"r"(taddr + SFA_COL + slot * 4), "l"(desc_plain(sF, 128, 128)) : "memory");
            asm volatile("tcgen05.cp.cta_group::1.32x128b.warpx4 [%0], %1;" ::"r"(taddr + SFB_COL + slot * 8), "l"(desc_plain(sF + 512, 128, 128)) : "memory");
            if (BN == 256)
              asm volatile("tcgen05.cp.cta_group::1.32x128b.warpx4 [%0], %1;" ::"r"(taddr + SFB_COL + slot * 8 + 4), "l"(desc_plain(sF + 1024, 128, 128)) : "memory");
          }
          const uint32_t sf_slot = UNIT ? 0 : slot;
#pragma unroll
          for (int kb = 0; kb < 4; kb++) {
            const uint64_t da = desc_sw128(sA + kb * 32), db = desc_sw128(sB + kb * 32);
            // block-scaled instruction descriptor: B scale id [4,6), E4M3 x E4M3, N>>3 [17,23), E8M0 scales (bit 23), M>>7 [27,29), A scale id [29,31)
            const uint32_t idesc = ((uint32_t)kb << 4) | ((uint32_t)(BN >> 3) << 17) | (1u << 23) | ((uint32_t)(BM >> 7) << 27) | ((uint32_t)kb << 29);
            const uint32_t acc = (kt > 0 || kb > 0) ? 1u : 0u;
            asm volatile("{\n.reg .pred p;\nsetp.ne.u32 p, %6, 0;\n"
                         "tcgen05.mma.cta_group::1.kind::mxf8f6f4.block_scale.scale_vec::1X [%0], %1, %2, %3, [%4], [%5], p;\n}"
                         ::"r"(taddr), "l"(da), "l"(db), "r"(idesc), "r"(taddr + SFA_COL + sf_slot * 4), "r"(taddr + SFB_COL + sf_slot * 8), "r"(acc) : "memory");
          }
          asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(s32(&bar_empty[slot])) : "memory");
        }
        if (ok) asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(s32(&bar_acc_full)) : "memory");
      }
      if (!ok) {     // leave nothing in flight before the tensor memory is given back
        asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(s32(&bar_drain)) : "memory");
#pragma unroll 1
        for (int i = 0; i < SPIN; i++) {
          uint32_t done;
          asm volatile("{\n.reg .pred p;\nmbarrier.try_wait.parity.shared::cta.b64 p, [%1], 0;\nselp.u32 %0, 1, 0, p;\n}" : "=r"(done) : "r"(s32(&bar_drain)) : "memory");
          if (done) break;
        }
      }
    }
  } else {
    // ---------------------------------------------------------------- epilogue: accumulator row r = tensor-memory lane r
    // Four warps per 32-lane sub-partition (a warp reaches only the lanes of sub-partition warp % 4), 64 columns each.  A warp brings
    // its columns into registers with two loads in flight and ONE wait, releases the accumulator, and only then does its arithmetic
    // and stores: the next tile's MMAs wait for one tensor-memory round trip, not for the epilogue.
    const int sub = warp & 3, cq = warp < EPI_WARPS ? 0 : 1 + (warp - (EPI_WARPS + LOAD_WARPS + 1)) / 4;      // column quarter 0..3
    uint32_t tile_i = 0;
    // the accumulator has been read: one arrival per warp
    auto release = [&]() {
      asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
      __syncwarp();
      if (lane == 0) arrive(s32(&bar_acc_empty));
    };
#pragma unroll 1
    for (int t = blockIdx.x; t < n_tiles; t += gridDim.x, tile_i++) {
      const int mt = t / tiles_n, n0 = (t % tiles_n) * BN, grp = group_of(mt), m0 = s_off[grp] + (mt - s_tile[grp]) * BM;
      int few = 0;                      // rows of a tile of FEW_ROWS
      if constexpr (OUT == OUT_SWIGLU && BN == 64) if (a_rows == FEW_ROWS) few = min(min(ends ? ends[grp] : off[grp + 1], m_total) - m0, FEW_ROWS);
      if (!wait_bar(s32(&bar_acc_full), tile_i & 1, abort_flag)) break;
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      if (BN < 256 && (cq * (OUT == OUT_SWIGLU ? 32 : 64) >= (OUT == OUT_SWIGLU ? BN / 2 : BN) || (BN == 64 && sub * 32 >= a_rows))) {      // no columns or no rows for this warp
        release();
        continue;
      }
      const uint32_t ta = taddr + ((uint32_t)(sub * 32) << 16);
      const size_t row = (size_t)(m0 + sub * 32 + lane);
      uint32_t v0[32], v1[32];
      if constexpr (OUT == OUT_SWIGLU) {
        // Fused activation between the expert GEMMs: the B rows of this tile are 128 gate rows followed by the 128 matching up rows
        // (the caller interleaves them so), so accumulator columns c and 128 + c belong together.  A thread holds 32 consecutive
        // outputs of its row = one MX block: bf16-round gate and up (what the unfused path stores), silu(gate) * up in fp32,
        // bf16-round, block exponent from the amax, E4M3 codes -- the arithmetic of swiglu_quant_kernel, with no trip through HBM.
        tmem_ld32(ta + cq * 32, v0); tmem_ld32(ta + BN / 2 + cq * 32, v1);
        asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
        release();
        if (BN == 64 && few) swiglu_quant_few(v0, v1, reinterpret_cast<float*>(sm_raw + (ring - s32(sm_raw)) + STAGES * STAGE_BYTES), act_q, act_e8, (size_t)m0, few, n >> 1, n0 >> 1);
        else swiglu_quant_store(v0, v1, act_q, act_e8, row, n >> 1, (n0 >> 1) + cq * 32);
      } else {
        tmem_ld32(ta + cq * 64, v0); tmem_ld32(ta + cq * 64 + 32, v1);
        asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
        release();
        // Results leave through this warp's staging rows (32 rows x 128 bytes, packet p of row r at p ^ (r & 7): conflict-free both ways), which are in the
        // 128-byte-swizzle layout a tiled tensor-map store reads: one copy of whole 128-byte row segments.  Rows past the tensor's last are not written.
        unsigned char* const stg = sm_raw + (ring - s32(sm_raw)) + STAGES * STAGE_BYTES + (warp < EPI_WARPS ? warp : warp - (LOAD_WARPS + 1)) * 4096;
        auto packet = [&](int p) { return stg + lane * 128 + ((p ^ (lane & 7)) << 4); };
        auto send = [&](int column) {
          asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
          __syncwarp();
          if (lane == 0) {
            asm volatile("cp.async.bulk.tensor.2d.global.shared::cta.tile.bulk_group [%0, {%1, %2}], [%3];"
                         ::"l"(&tm_c), "r"(column), "r"(m0 + sub * 32), "r"(s32(stg)) : "memory");
            asm volatile("cp.async.bulk.commit_group;" ::: "memory");
            asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");      // the rows may be overwritten
          }
          __syncwarp();
        };
        if constexpr (OUT == OUT_SCALED) {
          // (each thread storing its own row, 16 bytes of 32 rows an instruction: 47.7 us for the call of 1000 x 4096 x 4096 with fp32 results, 45.0 so)
          const float w = *so.fw, xf = *so.fx;
          const int col = n0 + cq * 64;
          if (m0 + sub * 32 < so.rows) {
            float b[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
            for (int j = 0; j < 64; j += 4) {
              const uint32_t* v = j < 32 ? v0 + j : v1 + (j - 32);
              if (so.bias) { const float4 b4 = __ldg(reinterpret_cast<const float4*>(so.bias + col + j)); b[0] = b4.x; b[1] = b4.y; b[2] = b4.z; b[3] = b4.w; }
              float o[4];
#pragma unroll
              for (int q = 0; q < 4; q++) {
                o[q] = __fmul_rn(__fmul_rn(__uint_as_float(v[q]), w), xf);      // y * w_scale * x_scale, in that order
                if (so.bias) o[q] = __fadd_rn(o[q], b[q]);
              }
              if (so.y_f16) {
                const __half2 h[2] = {__floats2half2_rn(o[0], o[1]), __floats2half2_rn(o[2], o[3])};
                *reinterpret_cast<uint2*>(packet(j >> 3) + (j & 4) * 2) = *reinterpret_cast<const uint2*>(h);
              } else {
                *reinterpret_cast<float4*>(packet((j >> 2) & 7)) = make_float4(o[0], o[1], o[2], o[3]);
                if (j == 28) send(col);
              }
            }
            send(so.y_f16 ? col : col + 32);
          }
        } else if constexpr (OUT == OUT_F32) {      // unrounded sums (the per-tensor FP8 linear scales them afterwards): each thread stores its own row
          float4* o4 = reinterpret_cast<float4*>(reinterpret_cast<float*>(c) + row * n + n0 + cq * 64);
#pragma unroll
          for (int j = 0; j < 8; j++) {
            o4[j] = make_float4(__uint_as_float(v0[4 * j]), __uint_as_float(v0[4 * j + 1]), __uint_as_float(v0[4 * j + 2]), __uint_as_float(v0[4 * j + 3]));
            o4[8 + j] = make_float4(__uint_as_float(v1[4 * j]), __uint_as_float(v1[4 * j + 1]), __uint_as_float(v1[4 * j + 2]), __uint_as_float(v1[4 * j + 3]));
          }
        } else {
          // row `lane`, 64 columns = eight 16-byte packets
#pragma unroll
          for (int p8 = 0; p8 < 8; p8++) {
            uint4 pk;
            __nv_bfloat162* h = reinterpret_cast<__nv_bfloat162*>(&pk);
#pragma unroll
            for (int q = 0; q < 4; q++) {
              const int j = p8 * 8 + 2 * q;
              h[q] = j < 32 ? __floats2bfloat162_rn(__uint_as_float(v0[j]), __uint_as_float(v0[j + 1]))
                            : __floats2bfloat162_rn(__uint_as_float(v1[j - 32]), __uint_as_float(v1[j - 31]));
            }
            *reinterpret_cast<uint4*>(packet(p8)) = pk;
          }
          send(n0 + cq * 64);
        }
      }
    }
    if (lane == 0) asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");      // this warp's stores have left before the CTA does
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (warp == EPI_WARPS + LOAD_WARPS) {
    __syncwarp();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(TMEM_COLS) : "memory");
  }
}

}  // namespace

extern "C" int b200q_mx_status_read_clear(int* status) {
  if (!status) return B200Q_ERR_BAD_ARG;
  int zero = 0;
  B200Q_CHECK_CUDA(cudaMemcpyFromSymbol(status, g_mx_status, sizeof(int)));
  B200Q_CHECK_CUDA(cudaMemcpyToSymbol(g_mx_status, &zero, sizeof(int)));
  int ep = 0;
  const int rc = b200q_ep_status_take(&ep);       // the exchange kernels around the expert GEMMs report through the same word
  if (rc) return rc;
  if (*status == 0) *status = ep;
  return B200Q_OK;
}

// [rows, k] elements, row-major -> tiled tensor map with boxes of `box_rows` rows x 128 bytes in the 128-byte-swizzle shared-memory layout.
// The encoder is a driver entry point; it is looked up through the runtime so that the library links against cudart only.
static int make_map(CUtensorMap* tm, const void* base, uint64_t rows, uint64_t k, uint32_t box_rows, CUtensorMapDataType type = CU_TENSOR_MAP_DATA_TYPE_UINT8, int size = 1) {
  typedef CUresult (*encode_fn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*, const cuuint32_t*,
                                const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
  static encode_fn fn = nullptr;
  if (!fn) {
    void* p = nullptr;
    cudaDriverEntryPointQueryResult q;
    B200Q_CHECK_CUDA(cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q));
    if (!p || q != cudaDriverEntryPointSuccess) return B200Q_ERR_UNSUPPORTED;
    fn = (encode_fn)p;
  }
  const cuuint64_t dims[2] = {k, rows}, strides[1] = {k * size};
  const cuuint32_t box[2] = {(cuuint32_t)(128 / size), box_rows}, estr[2] = {1, 1};
  const CUresult r = fn(tm, type, 2, const_cast<void*>(base), dims, strides, box, estr,
                        CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  return r == CUDA_SUCCESS ? B200Q_OK : B200Q_ERR_BAD_ARG;
}

// How wide a tile: the one whose waves over the SMs, each as long as the operand bytes of a K step, take the least; the widest among equals.  FP8 Linear 4096 x 4096, us a call
// with tiles of 256 columns and so: 1 row 33.3 / 20.3, 300 rows 37.5 / 23.1, 2000 rows 74.1 / 56.2 (there the width is the same, and all of the gain, as 2 to 6 us of the
// others, is the block scales that need not be brought in); 6144 -> 1024, 500 rows 59.4 / 42.1.  Expert layer 2048 x 1024, 64 experts top 8, one token 41.9 / 36.9.
static int tile_columns(int row_tiles, int n, int n_sm) {
  int best = 0;
  long long least = 0;
  for (int bn : {256, 128, 64}) {
    const long long tiles = (long long)row_tiles * (n / bn), t = (tiles + n_sm - 1) / n_sm * (BM + bn);
    if (!best || t < least) { best = bn; least = t; }
  }
  return best;
}
typedef decltype(&grouped_mxfp8_tc_kernel<OUT_BF16, 256>) GroupedKernel;
template <int BN> static GroupedKernel pick_out(int out) {
  return out == OUT_SWIGLU ? grouped_mxfp8_tc_kernel<OUT_SWIGLU, BN> : out == OUT_SCALED ? grouped_mxfp8_tc_kernel<OUT_SCALED, BN>
         : out == OUT_F32 ? grouped_mxfp8_tc_kernel<OUT_F32, BN> : grouped_mxfp8_tc_kernel<OUT_BF16, BN>;
}
static GroupedKernel pick_kernel(int out, int bn) { return bn == 256 ? pick_out<256>(out) : bn == 128 ? pick_out<128>(out) : pick_out<64>(out); }

// row_tiles: about how many tiles of 128 rows there are (0: all of m_total); few_rows: no group has more than FEW_ROWS.
static int grouped_launch(const void* a_q, const void* a_e8, const void* b_q, const void* b_e8, const int32_t* off, int n_experts, int m_total, int n, int k,
                          void* c_bf16, void* act_q, void* act_e8, void* stream, bool c_f32 = false, ScaledOut so = ScaledOut{}, bool pdl = false, const int32_t* ends = nullptr,
                          int row_tiles = 0, bool few_rows = false) {
  if (!a_q || !b_q || (!so.fw && (!a_e8 || !b_e8)) || !off || (!c_bf16 && !act_q) || n_experts <= 0 || m_total <= 0 || n <= 0 || k <= 0) return B200Q_ERR_BAD_ARG;
  if (act_q && (!act_e8 || (((uintptr_t)act_q) & 15))) return B200Q_ERR_BAD_ARG;
  if (m_total % 256 || n % BN_MAX || k % BK) return B200Q_ERR_BAD_SHAPE;       // the reference asks M % 256 == N % 256 == K % 128 == 0 (moe_gemm.py:120)
  if (n_experts > MAX_EXPERTS) return B200Q_ERR_UNSUPPORTED;
  if (((uintptr_t)a_q | (uintptr_t)b_q | (uintptr_t)c_bf16) & 15 || ((uintptr_t)a_e8 | (uintptr_t)b_e8) & 3) return B200Q_ERR_MISALIGNED;
  const int out = act_q ? OUT_SWIGLU : so.fw ? OUT_SCALED : c_f32 ? OUT_F32 : OUT_BF16;
  const int dev = b200q_current_device(), n_sm = b200q_sm_count();
  if (dev < 0 || n_sm <= 0) return B200Q_ERR_CUDA;
  if (row_tiles <= 0 || row_tiles > m_total / BM) row_tiles = m_total / BM;
  const int bn = tile_columns(row_tiles, n, n_sm);
  auto kernel = pick_kernel(out, bn);
  const int smem = bn == 256 ? Geo<256>::SMEM_BYTES : bn == 128 ? Geo<128>::SMEM_BYTES : Geo<64>::SMEM_BYTES;
  static PerDeviceFlag attr_set[4][3];
  PerDeviceFlag& flag = attr_set[out][bn == 256 ? 0 : bn == 128 ? 1 : 2];
  if (!flag.test(dev)) {
    B200Q_CHECK_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
    flag.set(dev);
  }
  const long long tiles = (long long)(m_total / BM) * (n / bn);
  const int grid = (int)(tiles < n_sm ? tiles : n_sm), a_rows = few_rows && bn == 64 ? FEW_ROWS : BM;
  alignas(64) CUtensorMap tm_a, tm_b, tm_c;
  memset(&tm_a, 0, sizeof(tm_a)); memset(&tm_b, 0, sizeof(tm_b)); memset(&tm_c, 0, sizeof(tm_c));
  int rc = B200Q_OK;
  if (out == OUT_SCALED) rc = so.y_f16 ? make_map(&tm_c, c_bf16, (uint64_t)so.rows, (uint64_t)n, 32, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 2)
                           : make_map(&tm_c, c_bf16, (uint64_t)so.rows, (uint64_t)n, 32, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 4);
  else if (out == OUT_BF16) rc = make_map(&tm_c, c_bf16, (uint64_t)m_total, (uint64_t)n, 32, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2);
  if (rc == B200Q_OK) rc = make_map(&tm_a, a_q, (uint64_t)m_total, (uint64_t)k, a_rows);
  if (rc == B200Q_OK) rc = make_map(&tm_b, b_q, (uint64_t)n_experts * n, (uint64_t)k, out == OUT_SWIGLU && bn < 256 ? bn / 2 : bn);
  if (rc != B200Q_OK) return rc;
  B200Q_CHECK_CUDA(launch_k(kernel, dim3(grid), dim3(THREADS), (size_t)smem, (cudaStream_t)stream, pdl, (const uint8_t*)a_q, (const uint8_t*)a_e8,
                            (const uint8_t*)b_q, (const uint8_t*)b_e8, off, n_experts, m_total, n, k, (__nv_bfloat16*)c_bf16, (uint8_t*)act_q, (uint8_t*)act_e8,
                            tm_a, tm_b, tm_c, so, ends, a_rows));
  return B200Q_OK;
}

// codes without block scales (the kernel has its own units)
int b200q_mx_gemm_scaled(const void* a_q, const void* b_q, const int32_t* off, int m_total, int n, int k, void* y, int y_dtype, int rows, const float* fw, const float* fx,
                         const float* bias, cudaStream_t st) {
  return grouped_launch(a_q, nullptr, b_q, nullptr, off, 1, m_total, n, k, y, nullptr, nullptr, st, true, ScaledOut{fw, fx, bias, rows, y_dtype == B200Q_F16}, true, nullptr,
                        (rows + BM - 1) / BM, rows <= FEW_ROWS);
}

// the expert layer's GEMMs (c_bf16: plain rows, else SwiGLU + requantise into act_q / act_e8), programmatic behind this library's kernels
// n_tokens x topk rows: an expert has a token once at most
int b200q_mx_gemm_chain(const void* a_q, const void* a_e8, const void* b_q, const void* b_e8, const int32_t* off, const int32_t* ends, int n_experts, int m_total, int n,
                        int k, void* c_bf16, void* act_q, void* act_e8, int n_tokens, int topk, cudaStream_t st) {
  const long long pairs = (long long)n_tokens * topk, tiles = n_tokens <= BM ? std::min<long long>(n_experts, pairs) : (pairs + BM - 1) / BM + n_experts / 2;
  return grouped_launch(a_q, a_e8, b_q, b_e8, off, n_experts, m_total, n, k, c_bf16, act_q, act_e8, st, false, ScaledOut{}, true, ends,
                        (int)std::min<long long>(tiles, m_total / BM), n_tokens <= FEW_ROWS);
}

extern "C" int b200q_grouped_mxfp8_gemm(const void* a_q, const void* a_e8, const void* b_q, const void* b_e8, const int32_t* off, int n_experts,
                                        int m_total, int n, int k, void* c_bf16, void* stream) {
  if (!c_bf16) return B200Q_ERR_BAD_ARG;
  return grouped_launch(a_q, a_e8, b_q, b_e8, off, n_experts, m_total, n, k, c_bf16, nullptr, nullptr, stream);
}

extern "C" int b200q_grouped_mxfp8_gemm_f32(const void* a_q, const void* a_e8, const void* b_q, const void* b_e8, const int32_t* off, int n_experts,
                                            int m_total, int n, int k, float* c_f32, void* stream) {
  if (!c_f32) return B200Q_ERR_BAD_ARG;
  return grouped_launch(a_q, a_e8, b_q, b_e8, off, n_experts, m_total, n, k, c_f32, nullptr, nullptr, stream, true);
}

extern "C" int b200q_grouped_mxfp8_gemm_swiglu(const void* a_q, const void* a_e8, const void* b_q, const void* b_e8, const int32_t* off, int n_experts,
                                               int m_total, int n, int k, void* act_q, void* act_e8, void* stream) {
  if (!act_q || !act_e8) return B200Q_ERR_BAD_ARG;
  return grouped_launch(a_q, a_e8, b_q, b_e8, off, n_experts, m_total, n, k, nullptr, act_q, act_e8, stream);
}
