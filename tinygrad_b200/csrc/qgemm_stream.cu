// Linear over many activation rows on packed Q4_0 / Q8_0 weights (prompts, batched rows):  Y[m, n] = X[m, k] W[n, k]^T
// (+ bias, + residual, or the SwiGLU product of interleaved gate / up rows).  Replaces `Linear.__call__` for T > 1
// (tinygrad/nn/__init__.py:177; prefill chunks of tinygrad/llm/model.py:464-481).
//
// Numerics: fp32 activations are split into fp16 halves x = xh + xl, the dequantised weight into w = wh + wl (wh the fp16 product of
// quant and scale, wl its exact remainder), and y = wh xh + wh xl + wl xh is accumulated in fp32 on the tensor cores: the fp32
// activation times the unrounded weight to about 2^-22.  fp16 activations take one pass with the fp16-rounded weight.
// A row of fp32 activations whose largest value lies outside [1, 2^15) is scaled by a power of two first, which its outputs give back: above that the halves
// overflow (a value past 65504 made a row of NaN), below it their absolute floor of 2^-25 shows against the row's values.  In between, and with `unsplit` everywhere
// below 2^15, the halves are those of b200q_qgemm, bit for bit.
//
// What bounds it: three fp16 tensor passes for many rows; for few rows the weight stream and the unpacking.  So
//  * weights are the MMA's A operand (128 rows per instruction) and the activation rows its N: any row count rounded up to 16 fills the
//    instruction, and up to 128 rows the products with a remainder (wh xl, wl xh) have an accumulator of their own;
//  * a tile is up to 256 weight rows (two accumulators, the whole of tensor memory) by up to 256 activation rows: every unpacked weight meets
//    256 rows and every activation byte 256 weight rows.  With 128 x 128 tiles the activation operand alone took 2.4x the L2 traffic
//    and every weight was unpacked once per 128 rows.  Up to 128 rows, and where tiles are few, a tile is 128 weight rows
//    (more tiles to share, smaller partial sums), and where its loop is long enough the weights of such a tile go through tensor memory (qgemm_tmem.cuh; the rule is
//    takes_tmem below: of fp32 rows up to 128);
//  * roles are separate warps: 16 unpack the weights (packed blocks by asynchronous copies, several ahead -> fp16 halves in a ring of
//    shared-memory slots), one thread brings activation tiles in by bulk copies, one issues the MMAs; nothing meets at a block barrier;
//  * the K x tile space is dealt to one CTA per SM in equal contiguous runs (stream-K): no last wave.  A tile that spans CTAs leaves fp32
//    partial sums in the workspace; the CTA that arrives last adds them in the order of K (bit-reproducible) and writes the result.
//    Nobody waits for another CTA.
// Every mbarrier wait is bounded: on expiry a status word is set, all roles leave, copies and MMAs in flight are drained.
#include "common.cuh"
#include "tc_common.cuh"
#include <cuda_bf16.h>
#include <algorithm>
#include <cstddef>

namespace {

constexpr int UNPACK_WARPS = 16, UNPACK_THREADS = UNPACK_WARPS * 32;
constexpr int WARP_COPY = UNPACK_WARPS, WARP_MMA = UNPACK_WARPS + 1;
constexpr int THREADS = (UNPACK_WARPS + 2) * 32;
constexpr int KSTEP = 32;                               // one quant block of K per step
constexpr int RING_BYTES = 224 * 1024, MAX_SLOTS = 6;   // shared memory: slots of unpacked weights + activations
// Packed blocks wait in shared memory, one 16 / 32-byte block and its scale per unpack thread and round, up to MAX_AHEAD rounds ahead.  A queue in
// registers that moves up by a block waits for the newest load every time: whatever its depth, a round took a trip to HBM (measured when every row count came through
// here, 8B gate / up: 45 rows 83 us, 70 so; 8 rows 79, 60).
constexpr int MAX_AHEAD = 4;
__host__ __device__ constexpr int ahead_bytes(int qt) { return UNPACK_THREADS * (qt == B200Q_Q4_0 ? 20 : 36); }
constexpr int MAX_NT = 256;                             // activation rows per tile
constexpr size_t COUNTER_BYTES = 4096;                  // one arrival counter per CTA (a split tile is counted at the CTA that holds its head)

struct StreamParams {
  const uint8_t* w;
  const unsigned char* xt;       // activation tiles (split_rows)
  const float* down;             // per activation row: what undoes its scaling (NULL: rows are not scaled)
  float* part;
  unsigned* counters;
  const __half* bias;
  const void* residual;
  void* y;
  long long units;               // tiles x K groups
  // Units are dealt in multiples of this: 1, or a whole tile where the caller wants it so (`unsplit`) or the workspace has no room for partial
  // sums.  With whole tiles every output is one running sum (remainders' products not apart either) in the order of b200q_qgemm: the same bits.
  int grain, unsplit;
  int tiles, m, n_out, kgroups, n_row_tiles, nt, tok_tiles, slots, ahead, y_f16, silu_mul;
  int dump, d_cols;              // qgemm_tmem.cuh: where whole tiles wait in shared memory (0: nowhere), tensor-memory columns of the accumulators
};

// ---- activations: fp32 (or fp16) rows, optionally RMS-normed, -> fp16 halves as the tensor core reads them ---------------------
// workspace: per activation tile of nt rows and K step of 32: [4 chunks of 8 columns][nt rows hi | nt rows lo][16 bytes], contiguous, so
// that a step's operand is one bulk copy.  Element order inside a chunk: [0,2,1,3,4,6,5,7], the order the weight unpack delivers.
// One CTA: 8 rows (a core matrix) x a stretch of columns; a row's chunk is 32 bytes in, 16 + 16 bytes out, 8 rows make 128 contiguous bytes.
// What is asked of a whole row (its mean square for the norm, its largest value for the scale) the CTAs of a row's stretches share as a cluster; stretches of up
// to 2048 columns are read once and kept in registers, so rows that short need no cluster.  A prompt of 45 on 16 8B-shaped blocks when that took 3734 us (3080 since its
// weights go through tensor memory): 477 us more with rows read twice, in clusters from 2048 columns on, 3170 more with every CTA reading its whole rows (806 for the
// mean square alone, without a scale).  Prompts on 384- to
// 1024-wide models take 2 to 5 % more than without a scale: the reduction in front of the stores, about half a microsecond a launch.
constexpr int SPLIT_THREADS = 256, SPLIT_HOLD = 8;

__device__ __forceinline__ void load_chunk(const float* row, int k, float (&f)[8]) {
  const float4 a = *reinterpret_cast<const float4*>(row + k), b = *reinterpret_cast<const float4*>(row + k + 4);
  f[0] = a.x; f[1] = a.y; f[2] = a.z; f[3] = a.w; f[4] = b.x; f[5] = b.y; f[6] = b.z; f[7] = b.w;
}
__device__ __forceinline__ void weigh_chunk(float (&f)[8], const uint4& nw, float& ss, float& amax) {
  const __half2* h = reinterpret_cast<const __half2*>(&nw);
#pragma unroll
  for (int q = 0; q < 4; q++) {
    const float2 w = __half22float2(h[q]);
    ss = fmaf(f[2 * q], f[2 * q], fmaf(f[2 * q + 1], f[2 * q + 1], ss));
    f[2 * q] *= w.x; f[2 * q + 1] *= w.y;
    amax = fmaxf(amax, fmaxf(fabsf(f[2 * q]), fabsf(f[2 * q + 1])));
  }
}

template <typename T, bool CLUSTER>
__global__ void __launch_bounds__(SPLIT_THREADS) split_rows_kernel(const T* __restrict__ x, const __half* __restrict__ norm_w, float eps, int m, int n_in,
                                                                   int kgroups, int nt, int chunks_per_cta, unsigned char* __restrict__ xt,
                                                                   unsigned* __restrict__ counters, int n_counters, float* __restrict__ down, float lowest) {
  constexpr bool F32 = sizeof(T) == 4;
  constexpr int STEP = SPLIT_THREADS / 8;                                 // chunks of a row in hand at once
  pdl_wait();
  pdl_launch_dependents();
  const int tid = threadIdx.x;
  if (blockIdx.x == 0 && blockIdx.y == 0)
    for (int i = tid; i < n_counters; i += SPLIT_THREADS) counters[i] = 0;
  const int r = tid & 7, row = blockIdx.x * 8 + r;                       // row within the padded rows of all tiles
  const int tile = row / nt, in_tile = row - tile * nt;
  const int n_chunks = kgroups * 16, c0 = blockIdx.y * chunks_per_cta + (tid >> 3), c1 = min(n_chunks, (int)(blockIdx.y + 1) * chunks_per_cta);
  const int live = row < m ? n_in : 0;                                    // columns the row has
  const T* src = x + (size_t)row * n_in;
  const size_t row_bytes = (F32 ? 2 : 1) * (size_t)nt * 16;               // one chunk of a step
  unsigned char* dst = xt + (size_t)tile * n_chunks * row_bytes + (size_t)in_tile * 16;
  if constexpr (!F32) {
    for (int c = c0; c < c1; c += STEP) {
      uint4 raw = make_uint4(0, 0, 0, 0);
      if (c * 8 < live) raw = *reinterpret_cast<const uint4*>(src + c * 8);
      *reinterpret_cast<uint4*>(dst + (size_t)c * row_bytes) =
          make_uint4(prmt(raw.x, raw.y, 0x5410u), prmt(raw.x, raw.y, 0x7632u), prmt(raw.z, raw.w, 0x5410u), prmt(raw.z, raw.w, 0x7632u));
    }
  } else {
    __shared__ float red[SPLIT_THREADS / 32][8], red_max[SPLIT_THREADS / 32][8];
    const uint4 ones = make_uint4(0x3C003C00u, 0x3C003C00u, 0x3C003C00u, 0x3C003C00u);
    float held[SPLIT_HOLD][8], ss = 0.f, amax = 0.f;
    // SPLIT_HOLD chunks in flight; a stretch of at most so many per thread stays in registers until its row's factor is known
    const int first = blockIdx.y * chunks_per_cta;
    for (int b = first; b < c1; b += SPLIT_HOLD * STEP) {
      uint4 nw[SPLIT_HOLD];
#pragma unroll
      for (int i = 0; i < SPLIT_HOLD; i++) {
        if (b + i * STEP >= c1) break;                                    // (the same for all threads)
        const int c = b + i * STEP + (tid >> 3);
        nw[i] = ones;
#pragma unroll
        for (int q = 0; q < 8; q++) held[i][q] = 0.f;
        if (c < c1 && c * 8 < live) {
          load_chunk(src, c * 8, held[i]);
          if (norm_w) nw[i] = *reinterpret_cast<const uint4*>(norm_w + c * 8);
        }
      }
#pragma unroll
      for (int i = 0; i < SPLIT_HOLD; i++) {
        if (b + i * STEP >= c1) break;
        weigh_chunk(held[i], nw[i], ss, amax);
      }
    }
    ss += __shfl_xor_sync(0xffffffffu, ss, 8);
    ss += __shfl_xor_sync(0xffffffffu, ss, 16);
    amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, 8));
    amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, 16));
    if ((tid & 31) < 8) { red[tid >> 5][r] = ss; red_max[tid >> 5][r] = amax; }
    __syncthreads();
    float tot = 0.f;
#pragma unroll
    for (int i = 0; i < SPLIT_THREADS / 32; i++) { tot += red[i][r]; amax = fmaxf(amax, red_max[i][r]); }
    if (CLUSTER) {                                                        // with the other stretches of the rows
      __syncthreads();
      if (tid < 8) { red[0][r] = tot; red_max[0][r] = amax; }
      __syncwarp();
      cluster_sync();
      tot = 0.f;
      for (uint32_t c = 0; c < gridDim.y; c++) { tot += ld_cluster(s32(&red[0][r]), c); amax = fmaxf(amax, ld_cluster(s32(&red_max[0][r]), c)); }
    }
    float sc = 1.f;
    if (norm_w) { sc = 1.0f / sqrtf(tot / (float)n_in + eps); amax *= sc; }
    if (down) {
      float up = 1.f, inv = 1.f;
      if (!(amax >= lowest && amax < 32768.f)) pow2_scale(amax, up, inv);
      if (blockIdx.y == 0 && tid < 8) down[row] = inv;
      sc *= up;
    }
    auto store = [&](float (&f)[8], int c) {
      uint4 hi, lo;
#pragma unroll
      for (int q = 0; q < 8; q++) f[q] *= sc;
      split_chunk(f, hi, lo);
      *reinterpret_cast<uint4*>(dst + (size_t)c * row_bytes) = hi;
      *reinterpret_cast<uint4*>(dst + (size_t)c * row_bytes + (size_t)nt * 16) = lo;
    };
    if (chunks_per_cta <= SPLIT_HOLD * STEP) {
#pragma unroll
      for (int i = 0; i < SPLIT_HOLD; i++)
        if (c0 + i * STEP < c1) store(held[i], c0 + i * STEP);
    } else {
      for (int c = c0; c < c1; c += STEP) {
        float f[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
        uint4 nw = ones;
        if (c * 8 < live) {
          load_chunk(src, c * 8, f);
          if (norm_w) nw = *reinterpret_cast<const uint4*>(norm_w + c * 8);
        }
        weigh_chunk(f, nw, ss, amax);
        store(f, c);
      }
    }
    __syncwarp();
    if (CLUSTER) cluster_sync();                                          // nobody leaves while its sums are being read
  }
}

// ---- the product ---------------------------------------------------------------------------------------------------------------
struct Shared {                       // barriers and small words (static shared memory)
  uint64_t full[MAX_SLOTS], empty[MAX_SLOTS], acc_full, acc_empty, stored, counted, drained;
  uint32_t tmem, last;
  int abort;
};

// Barriers are named by their shared-memory address, taken once (`sb` = the address of the Shared block) and kept in a register.
#define BAR(sb, member) ((sb) + (uint32_t)offsetof(Shared, member))
__device__ __forceinline__ uint32_t pinned(uint32_t v) { asm volatile("" : "+r"(v)); return v; }

__device__ __forceinline__ void bar_init(uint32_t bar, int n) { asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(n)); }
__device__ __forceinline__ void bar_arrive(uint32_t bar) { asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory"); }
// Bounded wait: false once another role has given up, or when the time is over (then the others are told).
__device__ __forceinline__ bool bar_wait(uint32_t sb, uint32_t bar, uint32_t parity) {
  for (int i = 0; i < (1 << 20); i++) {
    uint32_t ok, gone;
    asm volatile("{\n.reg .pred p;\nmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2, %3;\nselp.u32 %0, 1, 0, p;\n}"
                 : "=r"(ok) : "r"(bar), "r"(parity), "r"(2000) : "memory");
    if (ok) return true;
    asm volatile("ld.volatile.shared::cta.u32 %0, [%1];" : "=r"(gone) : "r"(BAR(sb, abort)) : "memory");
    if (gone) return false;
  }
  asm volatile("st.volatile.shared::cta.u32 [%0], 1;" ::"r"(BAR(sb, abort)) : "memory");
  atomicExch(&g_tc_status, 1);
  return false;
}
__device__ __forceinline__ void commit(uint32_t bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar) : "memory");
}
// descriptors as {low word, common high word}: a step's operands differ in the start address alone
__device__ __forceinline__ void mma(uint32_t d, uint32_t a_lo, uint32_t b_lo, uint32_t hi, uint32_t idesc, uint32_t acc) {
  asm volatile("{\n.reg .pred p;\n.reg .b64 a, b;\nmov.b64 a, {%1, %3};\nmov.b64 b, {%2, %3};\nsetp.ne.u32 p, %5, 0;\n"
               "tcgen05.mma.cta_group::1.kind::f16 [%0], a, b, %4, p;\n}"
               ::"r"(d), "r"(a_lo), "r"(b_lo), "r"(hi), "r"(idesc), "r"(acc) : "memory");
}
__device__ __forceinline__ void st_shared(uint32_t a, const uint4& v) {
  asm volatile("st.shared::cta.v4.u32 [%0], {%1,%2,%3,%4};" ::"r"(a), "r"(v.x), "r"(v.y), "r"(v.z), "r"(v.w) : "memory");
}
constexpr int EC = 8;                                   // accumulator columns (activation rows) a thread of the epilogue takes at a time
__device__ __forceinline__ void ld_tmem(uint32_t a, uint32_t (&v)[EC]) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
               : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]) : "r"(a));
}

// unit range of CTA c (in whole grains), and the CTA that holds a unit (grain 1: tiles are split only then)
__device__ __forceinline__ long long first_unit(long long c, const StreamParams& p, int g) { return c * (p.units / p.grain) / g * p.grain; }
// Where CTA c leaves its part of a split tile.  Along the units either the CTA or the tile (or both) goes up by one from part to part, so
// c + tile is a number of its own for each; with more tiles than CTAs, two places per CTA (its first and its last part) take less room.
__device__ __forceinline__ size_t part_slot(const StreamParams& p, int c, int tile, bool head) {
  return p.tiles < (int)gridDim.x ? (size_t)(c + tile) : (size_t)(2 * c + (head ? 1 : 0));
}
__device__ __forceinline__ int cta_of(long long unit, long long units, int g) { return (int)(((unit + 1) * g - 1) / units); }

// N consecutive activation rows of one output column (weight row) `feat`
template <int N> __device__ __forceinline__ void store_outputs(const StreamParams& p, float (&v)[N], int feat, int tok0, int lane) {
  if (p.down)
#pragma unroll
    for (int j = 0; j < N; j += 4) {
      const float4 d = *reinterpret_cast<const float4*>(p.down + tok0 + j);
      v[j] *= d.x; v[j + 1] *= d.y; v[j + 2] *= d.z; v[j + 3] *= d.w;
    }
  if (p.silu_mul) {
    // gate rows sit in lanes with bit 3 clear, the matching up rows 8 lanes on: each of a pair takes every other activation row
    const bool gate = !(lane & 8);
    const int col = (feat >> 4) * 8 + (feat & 7), n_y = p.n_out >> 1;
#pragma unroll
    for (int j = 0; j < N; j += 2) {
      const float other = __shfl_xor_sync(0xffffffffu, gate ? v[j + 1] : v[j], 8);
      const float g = gate ? v[j] : other, u = gate ? other : v[j + 1], o = (g / (1.f + expf(-g))) * u;
      const int tok = tok0 + j + (gate ? 0 : 1);
      if (tok < p.m && col < n_y) {
        const size_t at = (size_t)tok * n_y + col;
        if (p.y_f16) reinterpret_cast<__half*>(p.y)[at] = __float2half_rn(o); else reinterpret_cast<float*>(p.y)[at] = o;
      }
    }
    return;
  }
  if (feat >= p.n_out) return;
  const float b = p.bias ? __half2float(p.bias[feat]) : 0.f;
  float add[N];
#pragma unroll
  for (int j = 0; j < N; j++) {
    add[j] = b;
    if (p.residual && tok0 + j < p.m) {
      const size_t at = (size_t)(tok0 + j) * p.n_out + feat;
      add[j] += p.y_f16 ? __half2float(reinterpret_cast<const __half*>(p.residual)[at]) : reinterpret_cast<const float*>(p.residual)[at];
    }
  }
#pragma unroll
  for (int j = 0; j < N; j++)
    if (tok0 + j < p.m) {
      const size_t at = (size_t)(tok0 + j) * p.n_out + feat;
      if (p.y_f16) reinterpret_cast<__half*>(p.y)[at] = __float2half_rn(v[j] + add[j]); else reinterpret_cast<float*>(p.y)[at] = v[j] + add[j];
    }
}

// The 16 unpack warps read the accumulators of segment `seg` (K groups k0 .. k1 of `tile`) back.
template <int WT, bool F32>
__device__ __forceinline__ bool finish_segment(const StreamParams& p, Shared& sh, uint32_t sb, int seg, int tile, int k0, int k1) {
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, sub = warp & 3, q = warp >> 2;
  const int hf = WT == 256 ? q >> 1 : 0, part0 = WT == 256 ? q & 1 : q, parts = WT == 256 ? 2 : 4;
  const int tt = tile % p.tok_tiles, row = hf * 128 + sub * 32 + lane, feat = (tile / p.tok_tiles) * WT + row;
  const bool whole = k0 == 0 && k1 == p.kgroups, two_sums = WT == 128 && F32 && p.nt <= MAX_NT / 2 && !p.unsplit;
  const int G = gridDim.x, c = blockIdx.x;
  int c0 = c, n_seg = 1;
  if (!whole) {
    c0 = cta_of((long long)tile * p.kgroups, p.units, G);
    n_seg = cta_of((long long)(tile + 1) * p.kgroups - 1, p.units, G) - c0 + 1;
  }
  const size_t slot = (size_t)WT * p.nt;
  float* mine = p.part + part_slot(p, c, tile, c == c0) * slot + row * 4;      // [group of 4 columns][row][4]: a warp's store is 512 contiguous bytes
  if (!bar_wait(sb, BAR(sb, acc_full), seg & 1)) return false;
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t ta = sh.tmem + ((uint32_t)(sub * 32) << 16) + hf * 256;
  const int groups = p.nt / EC;
  for (int cg = part0; cg < groups; cg += parts) {
    uint32_t a[EC], b[EC];
    ld_tmem(ta + cg * EC, a);
    if (two_sums) ld_tmem(ta + p.nt + cg * EC, b);
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
    float v[EC];
#pragma unroll
    for (int j = 0; j < EC; j++) v[j] = two_sums ? __uint_as_float(a[j]) + __uint_as_float(b[j]) : __uint_as_float(a[j]);
    if (whole) store_outputs(p, v, feat, tt * p.nt + cg * EC, lane);
    else
#pragma unroll
      for (int j = 0; j < EC; j += 4) __stcg(reinterpret_cast<float4*>(mine + (size_t)(cg * EC + j) * WT), make_float4(v[j], v[j + 1], v[j + 2], v[j + 3]));
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncwarp();
  if (lane == 0) { bar_arrive(BAR(sb, acc_empty)); if (!whole) bar_arrive(BAR(sb, stored)); }
  if (whole) return true;
  // a CTA has at most two partial segments: its first and its last; `stored` / `counted` complete once for each
  const uint32_t par = c == c0 && first_unit(c, p, G) % p.kgroups != 0 ? 1 : 0;
  if (tid == 0 && bar_wait(sb, BAR(sb, stored), par)) {
    __threadfence();
    const unsigned old = atomicAdd(p.counters + c0, 1u);
    const bool last = old == (unsigned)n_seg - 1;
    if (last) p.counters[c0] = 0;
    sh.last = last;
    __threadfence();
    bar_arrive(BAR(sb, counted));
  }
  if (!bar_wait(sb, BAR(sb, counted), par)) return false;
  if (!*reinterpret_cast<volatile uint32_t*>(&sh.last)) return true;
  const float* from = p.part + row * 4;
  for (int cg = part0; cg < groups; cg += parts) {
    float v[EC];
#pragma unroll
    for (int j = 0; j < EC; j++) v[j] = 0.f;
#pragma unroll 2
    for (int s = 0; s < n_seg; s++) {
      const float* sp = from + part_slot(p, c0 + s, tile, s == 0) * slot + (size_t)cg * EC * WT;
#pragma unroll
      for (int j = 0; j < EC; j += 4) {
        const float4 f = __ldcg(reinterpret_cast<const float4*>(sp + (size_t)j * WT));
        v[j] += f.x; v[j + 1] += f.y; v[j + 2] += f.z; v[j + 3] += f.w;
      }
    }
    store_outputs(p, v, feat, tt * p.nt + cg * EC, lane);
  }
  return true;
}

}  // namespace
#include "qgemm_tmem.cuh"
namespace {

// the weights of one 32-wide block of a row as they come from memory
template <int QT> struct Raw;
template <> struct Raw<B200Q_Q4_0> { uint4 a; uint32_t d; };
template <> struct Raw<B200Q_Q8_0> { uint4 a, b; uint32_t d; };

template <int QT, int WT, bool F32>
__global__ void __launch_bounds__(THREADS, 1) qgemm_stream_kernel(const StreamParams p) {
  constexpr int TB = tile_bytes(QT), GROUPS = UNPACK_THREADS / WT, PER_UNIT = 4 / GROUPS;    // thread groups, each with its own steps of a K group
  constexpr int W_HALF = WT * KSTEP * 2, W_STEP = 2 * W_HALF;
  extern __shared__ __align__(128) unsigned char dyn[];
  __shared__ Shared sh;
  const uint32_t sb = pinned(s32(&sh)), ring = pinned(s32(dyn));
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int G = gridDim.x, c = blockIdx.x;
  const long long u0 = first_unit(c, p, G), u1 = first_unit(c + 1, p, G);
  const int nt = p.nt, slots = p.slots, x_rows = F32 ? 2 * nt : nt;
  const uint32_t x_step = (uint32_t)x_rows * 64, slot_bytes = W_STEP + x_step;      // a slot: one step's activations and weights
  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(s32(&sh.tmem)), "r"(WT == 256 ? 512 : 256) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  if (tid == 32) {
    // a slot is full when its unpack warps and the copy thread have arrived and the copy's bytes are there; one commit empties it
    for (int i = 0; i < MAX_SLOTS; i++) { bar_init(BAR(sb, full) + 8 * i, WT / 32 + 1); bar_init(BAR(sb, empty) + 8 * i, 1); }
    bar_init(BAR(sb, acc_full), 1); bar_init(BAR(sb, acc_empty), UNPACK_WARPS);
    bar_init(BAR(sb, stored), UNPACK_WARPS); bar_init(BAR(sb, counted), 1); bar_init(BAR(sb, drained), 1);
    sh.abort = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  pdl_launch_dependents();

  if (warp == WARP_COPY) {
    if (elect_one()) {
      pdl_wait();                                        // the activation tiles are the previous kernel's (generic stores, read by bulk copies here)
      asm volatile("fence.proxy.async.global;" ::: "memory");
      bool ok = true;
      int n = 0, slot = 0;                               // steps issued; ring position (counted, not divided: this thread's loop is the copies' pace)
      uint32_t par = 1;
      for (long long u = u0; u < u1 && ok;) {
        const int tile = (int)(u / p.kgroups), k0 = (int)(u - (long long)tile * p.kgroups), k1 = (int)min((long long)p.kgroups, k0 + u1 - u);
        const unsigned char* src = p.xt + ((size_t)(tile % p.tok_tiles) * p.kgroups + k0) * 4 * x_step;
        for (int s = 0; s < (k1 - k0) * 4; s++, n++, src += x_step) {
          if (!bar_wait(sb, BAR(sb, empty) + 8 * slot, par)) { ok = false; break; }
          const uint32_t dst = ring + slot * slot_bytes + W_STEP, bar = BAR(sb, full) + 8 * slot;
          asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(x_step) : "memory");
          for (uint32_t o = 0; o < x_step; o += 8192)   // several copies overlap where one is served slowly
            asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
                         ::"r"(dst + o), "l"(src + o), "r"(min(8192u, x_step - o)), "r"(bar) : "memory");
          if (++slot == slots) { slot = 0; par ^= 1; }
        }
        u += k1 - k0;
      }
      // Nothing may still be landing in shared memory when the CTA leaves.  After a failed wait a slot's unpack warps may never arrive, so its
      // barrier cannot tell; the copies are done long before the time that wait took, and one more is spent here.
      for (int j = max(0, n - slots); j < n; j++)
        if (!wait_bar(BAR(sb, full) + 8 * (j % slots), (j / slots) & 1)) break;
    }
  } else if (warp == WARP_MMA) {
    if (elect_one()) {
      bool ok = true;
      const bool two_sums = WT == 128 && F32 && nt <= MAX_NT / 2 && !p.unsplit;
      const uint32_t id = make_idesc(128, nt), lo = two_sums ? nt : 0;      // one shape, the remainders' products beside: see qgemm_tmem.cuh
      const uint32_t desc_hi = (uint32_t)(make_desc(0, 0, 128) >> 32);
      const uint32_t w_base = (ring >> 4) | ((uint32_t)WT << 16), x_base = ((ring + W_STEP) >> 4) | ((uint32_t)x_rows << 16);
      int seg = 0, slot = 0;
      uint32_t par = 0, x_lo = x_base, w_lo = w_base;
      for (long long u = u0; u < u1 && ok; seg++) {
        const int k0 = (int)(u % p.kgroups), k1 = (int)min((long long)p.kgroups, k0 + u1 - u);
        if (!bar_wait(sb, BAR(sb, acc_empty), (seg & 1) ^ 1)) { ok = false; break; }
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        const uint32_t tmem = sh.tmem;
        uint32_t acc = 0, acc_lo = two_sums ? 0 : 1;
        for (int s = (k1 - k0) * 4; s > 0; s--) {
          if (!bar_wait(sb, BAR(sb, full) + 8 * slot, par)) { ok = false; break; }
          asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
          // all MMAs of one accumulator back to back; with weights in shared memory an instruction of N <= 96 takes 40 to 57 cycles whatever its N, of 256 129
#pragma unroll
          for (int hf = 0; hf < WT / 128; hf++) {
            const uint32_t d = tmem + hf * 256;
#pragma unroll
            for (int kk = 0; kk < KSTEP / 16; kk++) {
              const uint32_t xh = x_lo + (kk >> 1) * (x_step >> 4) + (kk & 1) * 2 * x_rows;
              const uint32_t wh = w_lo + (kk >> 1) * (W_STEP >> 4) + hf * 128 + (kk & 1) * 2 * WT;
              mma(d, wh, xh, desc_hi, id, kk ? 1u : acc);
              if (F32) {
                mma(d + lo, wh, xh + nt, desc_hi, id, kk ? 1u : acc_lo);
                mma(d + lo, wh + (W_HALF >> 4), xh, desc_hi, id, 1u);
              }
            }
          }
          acc = acc_lo = 1;
          commit(BAR(sb, empty) + 8 * slot);
          x_lo += slot_bytes >> 4; w_lo += slot_bytes >> 4;
          if (++slot == slots) { slot = 0; par ^= 1; x_lo = x_base; w_lo = w_base; }
        }
        if (ok) commit(BAR(sb, acc_full));
        u += k1 - k0;
      }
      commit(BAR(sb, drained));                               // also on the way out after a failed wait: MMAs issued must be done before tensor memory goes back
      wait_bar(BAR(sb, drained), 0);
    }
  } else {
    // ------------------------------ unpack ------------------------------
    // Thread group `grp` takes the steps t = grp, grp + GROUPS, .. of every K group; a thread takes one weight row's block of 32.
    const int grp = tid / WT, r = tid % WT, h8 = (r >> 3) & 1, g = r & 7;
    // The block being fetched.  A weight row's K groups are contiguous, so within a tile the pointer only moves on.
    const int in_w = (h8 * (QT == B200Q_Q4_0 ? 32 : 64) + g * 4 + grp) * 16, in_d = TB - 128 + (2 * g * 4 + h8 * 2) * 2;
    int ft = (int)(u0 / p.kgroups), f_left = (int)min((long long)p.kgroups - (u0 - (long long)ft * p.kgroups), u1 - u0), fs = 0;
    int f_units = (int)(u1 - u0);                        // units still to fetch
    const uint8_t* fp = nullptr;
    auto set_tile = [&](int k0) {
      const int f_row = ft / p.tok_tiles * (WT / 16) + (r >> 4);
      fp = f_row < p.n_row_tiles ? p.w + ((size_t)f_row * p.kgroups + k0) * TB : nullptr;
    };
    set_tile((int)(u0 - (long long)ft * p.kgroups));
    // this thread's places among the waiting blocks (never read by another thread, so no barrier)
    constexpr uint32_t AHEAD = ahead_bytes(QT), SCALE_AT = UNPACK_THREADS * (QT == B200Q_Q4_0 ? 16 : 32);
    const uint32_t wait0 = ring + slots * slot_bytes, wait_end = wait0 + p.ahead * AHEAD;
    uint32_t wait_at = wait0;                            // the oldest waiting block
    auto request = [&](uint32_t at) {                    // copies the next block there; zeros past the last row tile or K group
      const bool in = fp && f_units > 0;
      const uint8_t* src = in ? fp : p.w;
      const uint32_t n16 = in ? 16u : 0u, n4 = in ? 4u : 0u;
      const int w_at = in_w + fs * GROUPS * 16;
      asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(at + tid * 16), "l"(src + (in ? w_at : 0)), "r"(n16) : "memory");
      if constexpr (QT == B200Q_Q8_0)
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(at + UNPACK_THREADS * 16 + tid * 16), "l"(src + (in ? w_at + 512 : 0)), "r"(n16) : "memory");
      asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(at + SCALE_AT + tid * 4), "l"(src + (in ? in_d + ((grp + fs * GROUPS) >> 1) * 8 : 0)), "r"(n4) : "memory");
      asm volatile("cp.async.commit_group;" ::: "memory");
      if (PER_UNIT == 1 || ++fs == PER_UNIT) {
        fs = 0; f_units--;
        if (in) fp += TB;
        if (--f_left == 0) { ft++; f_left = p.kgroups; set_tile(0); }
      }
    };
    auto collect = [&](Raw<QT>& q) {
      switch (p.ahead) {
        case 1: asm volatile("cp.async.wait_group 0;" ::: "memory"); break;
        case 2: asm volatile("cp.async.wait_group 1;" ::: "memory"); break;
        case 3: asm volatile("cp.async.wait_group 2;" ::: "memory"); break;
        default: asm volatile("cp.async.wait_group 3;" ::: "memory");
      }
      q.a = ld_shared4(wait_at + tid * 16);
      if constexpr (QT == B200Q_Q8_0) q.b = ld_shared4(wait_at + UNPACK_THREADS * 16 + tid * 16);
      uint32_t d;
      asm volatile("ld.shared.u32 %0, [%1];" : "=r"(d) : "r"(wait_at + SCALE_AT + tid * 4) : "memory");
      q.d = grp & 1 ? d >> 16 : d & 0xFFFFu;
    };
    for (int d = 0; d < p.ahead; d++) request(wait0 + d * AHEAD);
    pdl_wait();                                          // the epilogue reads and writes what earlier kernels touched
    // One block: wait for its slot, unpack, hand over, ask for the block DEPTH further on.
    int slot = grp;                                      // ring position and its phase; the thread groups take turns
    uint32_t par = 1;
    bool ok = true;
    auto unpack = [&]() {
      ok = ok && bar_wait(sb, BAR(sb, empty) + 8 * slot, par);
      Raw<QT> q;
      collect(q);
      const uint32_t dst = ring + slot * slot_bytes + r * 16;
      const uint32_t d2 = q.d | (q.d << 16);
      uint4 hi[4], lo[4];
      if constexpr (QT == B200Q_Q4_0) {
        uint32_t v[4][4];
        q4_word(q.a.x, v[0]); q4_word(q.a.y, v[1]); q4_word(q.a.z, v[2]); q4_word(q.a.w, v[3]);
#pragma unroll
        for (int i = 0; i < 4; i++) {
          const int a = (i & 1) * 2, b = (i >> 1) * 2;      // chunk i: words a, a + 1; low or high nibbles
          const uint32_t r4[4] = {v[a][b], v[a][b + 1], v[a + 1][b], v[a + 1][b + 1]};
          hi[i] = hi_lo(r4, d2, lo[i]);
        }
      } else {
        hi[0] = q8_core(q.a.x, q.a.y, d2, lo[0]); hi[1] = q8_core(q.a.z, q.a.w, d2, lo[1]);
        hi[2] = q8_core(q.b.x, q.b.y, d2, lo[2]); hi[3] = q8_core(q.b.z, q.b.w, d2, lo[3]);
      }
      if (ok) {
#pragma unroll
        for (int i = 0; i < 4; i++) {
          st_shared(dst + i * (WT * 16), hi[i]);
          if (F32) st_shared(dst + W_HALF + i * (WT * 16), lo[i]);
        }
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
      }
      __syncwarp();
      if (lane == 0) bar_arrive(BAR(sb, full) + 8 * slot);
      request(wait_at);
      if ((wait_at += AHEAD) == wait_end) wait_at = wait0;
      slot += GROUPS;
      if (slot >= slots) { slot -= slots; par ^= 1; }
    };
    // A segment's accumulators are read back only after the first LEAD blocks of the next one are unpacked: they fill the ring while the
    // MMAs still in the pipe complete.
    const int LEAD = slots / GROUPS;
    int done_tile = -1, done_k0 = 0, done_k1 = 0, seg = 0;
    long long u = u0;
    while (ok) {
      int tile = 0, k0 = 0, k1 = 0, left = 0;
      if (u < u1) {
        tile = (int)(u / p.kgroups); k0 = (int)(u - (long long)tile * p.kgroups); k1 = (int)min((long long)p.kgroups, k0 + u1 - u);
        left = (k1 - k0) * PER_UNIT;
      }
      const int lead = done_tile >= 0 ? min(left, LEAD) : left;
      // one instance of the unpack code: unrolled the loop took 1.6x the cycles per block (instruction fetch)
#pragma unroll 1
      for (int stop = left - lead;; stop = 0) {
#pragma unroll 1
        for (; left > stop && ok; left--) {
          unpack();
        }
        if (done_tile >= 0 && ok) {
          ok = finish_segment<WT, F32>(p, sh, sb, seg++, done_tile, done_k0, done_k1);
          done_tile = -1;
        } else break;
      }
      if (u >= u1) break;
      done_tile = tile; done_k0 = k0; done_k1 = k1;
      u += k1 - k0;
    }
    asm volatile("cp.async.wait_group 0;" ::: "memory");      // nothing may still be landing when the CTA leaves
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (warp == 0) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(sh.tmem), "r"(WT == 256 ? 512 : 256) : "memory");
}

// ---- one fp32 row -----------------------------------------------------------------------------------------------------------------
// What stands between two GEMMs of a one-token step of a mixture-of-experts model, in one CTA: the weighted sum of the experts' outputs and its residual add (in.y), the
// RMSNorm, and the split halves of the row (the other rows of its tile are columns of the product that nobody reads).  Values and their order are those of
// combine8_kernel, rmsnorm_rows_kernel and split_rows_kernel, bit for bit: an expert's choice and its E4M3 codes turn a last-bit difference into a visible one.
constexpr int ROW_THREADS = 256;
__global__ void __launch_bounds__(ROW_THREADS) prepare_row_kernel(const b200q_row_input in, int n_in, int kgroups, int nt, unsigned char* __restrict__ xt, float* __restrict__ down) {
  extern __shared__ __align__(16) float row_s[];
  __shared__ float red[ROW_THREADS / 32];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  pdl_launch_dependents();
  pdl_wait();
  for (int c = tid * 8; c < n_in; c += ROW_THREADS * 8) {
    float f[8];
    load_chunk(in.x, c, f);
    if (in.y) {
      const __nv_bfloat16* y = reinterpret_cast<const __nv_bfloat16*>(in.y);
      float acc[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
      for (int j0 = 0; j0 < in.k; j0 += 4) {
        uint4 u[4];
#pragma unroll
        for (int j = 0; j < 4; j++) if (j0 + j < in.k) u[j] = *reinterpret_cast<const uint4*>(y + (size_t)in.dest_row[j0 + j] * n_in + c);
#pragma unroll
        for (int j = 0; j < 4; j++) {
          if (j0 + j < in.k) {
            const float w = in.weights[j0 + j];
            const uint32_t b[4] = {u[j].x, u[j].y, u[j].z, u[j].w};
#pragma unroll
            for (int i = 0; i < 4; i++) { acc[2 * i] += w * __uint_as_float(b[i] << 16); acc[2 * i + 1] += w * __uint_as_float(b[i] & 0xFFFF0000u); }
          }
        }
      }
#pragma unroll
      for (int i = 0; i < 8; i++) f[i] += __bfloat162float(__float2bfloat16_rn(acc[i]));
      *reinterpret_cast<float4*>(in.x + c) = make_float4(f[0], f[1], f[2], f[3]);
      *reinterpret_cast<float4*>(in.x + c + 4) = make_float4(f[4], f[5], f[6], f[7]);
    }
    *reinterpret_cast<float4*>(row_s + c) = make_float4(f[0], f[1], f[2], f[3]);
    *reinterpret_cast<float4*>(row_s + c + 4) = make_float4(f[4], f[5], f[6], f[7]);
  }
  __syncthreads();
  float sc = 1.f;
  if (in.norm_w) {
    float ss = 0.f;
    for (int i = tid; i < n_in; i += ROW_THREADS) { const float v = row_s[i]; ss += v * v; }
    ss = warp_sum(ss);
    if (lane == 0) red[warp] = ss;
    __syncthreads();
    float tot = 0.f;
    for (int i = 0; i < ROW_THREADS / 32; i++) tot += red[i];
    sc = 1.0f / sqrtf(tot / (float)n_in + in.eps);
    __syncthreads();
  }
  const __half* nw = reinterpret_cast<const __half*>(in.norm_w);
  auto value = [&](int c, float (&f)[8]) {
#pragma unroll
    for (int q = 0; q < 8; q++) f[q] = c + q < n_in ? (nw ? row_s[c + q] * sc * __half2float(nw[c + q]) : row_s[c + q]) : 0.f;
  };
  float amax = 0.f;
  for (int c = tid * 8; c < n_in; c += ROW_THREADS * 8) {
    float f[8];
    value(c, f);
#pragma unroll
    for (int q = 0; q < 8; q++) amax = fmaxf(amax, fabsf(f[q]));
  }
  amax = warp_max(amax);
  if (lane == 0) red[warp] = amax;
  __syncthreads();
#pragma unroll
  for (int i = 0; i < ROW_THREADS / 32; i++) amax = fmaxf(amax, red[i]);
  float up = 1.f, inv = 1.f;
  if (down) {
    if (!(amax < 32768.f)) pow2_scale(amax, up, inv);
    if (tid == 0) down[0] = inv;
  }
  const size_t row_bytes = (size_t)nt * 32;
  for (int c = tid; c < kgroups * 16; c += ROW_THREADS) {
    float f[8];
    uint4 hi, lo;
    value(c * 8, f);
#pragma unroll
    for (int q = 0; q < 8; q++) f[q] *= up;
    split_chunk(f, hi, lo);
    *reinterpret_cast<uint4*>(xt + (size_t)c * row_bytes) = hi;
    *reinterpret_cast<uint4*>(xt + (size_t)c * row_bytes + (size_t)nt * 16) = lo;
  }
}

// ---- launch --------------------------------------------------------------------------------------------------------------------
struct Plan { int nt, tok_tiles, wt; };
Plan make_plan(int m, int n_out, int n_sm) {
  Plan pl;
  pl.tok_tiles = ceil_div(m, MAX_NT);
  pl.nt = ceil_div(ceil_div(m, pl.tok_tiles), 16) * 16;      // equal tiles: 301 rows are 2 x 160, not 256 + 45
  // 128 weight rows a tile up to 128 activation rows (qgemm_tmem.cuh; 28672 x 4096, 128 rows: 256-row tiles through shared memory 87 us, 77), and where tiles of 256
  // are too few for the SMs: each is then split over several CTAs, the one that arrives last adds all parts alone, and halving the tile quarters what it reads.
  // 8B QKV (24 tiles), 256 rows: 75 -> 49 us, down (16) 117 -> 83; gate/up (112) 154 -> 142; 7B gate/up (148 tiles, hardly split) 142 -> 146.
  pl.wt = pl.nt <= 128 || (n_out > 0 && 5LL * ceil_div(n_out, 256) * pl.tok_tiles <= 4LL * n_sm) ? 128 : 256;
  return pl;
}
size_t tiles_bytes(const Plan& pl, int kgroups, bool f32) { return (size_t)pl.tok_tiles * pl.nt * kgroups * GROUP_ELEMS * (f32 ? 4 : 2); }
int slot_bytes(const Plan& pl, bool f32) { return pl.wt * KSTEP * 4 + pl.nt * (f32 ? 128 : 64); }
size_t align256(size_t n) { return (n + 255) & ~(size_t)255; }
size_t scale_bytes(const Plan& pl) { return align256((size_t)pl.tok_tiles * pl.nt * sizeof(float)); }

template <int QT, int WT, bool F32>
int launch_stream(const StreamParams& p, int grid, cudaStream_t st) {
  auto kern = qgemm_stream_kernel<QT, WT, F32>;
  static PerDeviceFlag attr;
  const int dev = b200q_current_device();
  if (dev < 0) return B200Q_ERR_CUDA;
  if (!attr.test(dev)) {
    B200Q_CHECK_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, RING_BYTES));
    attr.set(dev);
  }
  B200Q_CHECK_CUDA(launch_k(kern, dim3(grid), dim3(THREADS), (size_t)p.slots * slot_bytes({p.nt, p.tok_tiles, WT}, F32) + (size_t)p.ahead * ahead_bytes(QT), st, true, p));
  return B200Q_OK;
}

// Weights through tensor memory, or through shared memory (tiles of 128 weight rows; of fp32 rows at most 128 activation rows, 2 x 128 accumulator columns)?  The first wherever
// its faster loop runs long enough to pay for its longer way in and out.  Prompts on 1024-wide Q8_0 blocks (their Linears are 64 to 450 K groups, below 4 an SM): 62 tokens 976 us
// through tensor memory, through shared memory 873; 4096-wide (6 an SM and more): 1032, 1179.  45
// tokens: 1024-wide Q4_0 813, 853, Q8_0 872, 833; 2048-wide Q4_0 1086, 1121.  Above 64 rows the line is at 10 an SM: 4608 x 3584 (7), 128 rows 35.3 us, 32.0; 3584 x 18944 (28) 70,
// 74.  Tiles dealt to more than 8 CTAs (400 x 4096, 120 half-precision rows) are mostly the adding of their parts: 32 us, 25.
bool takes_tmem(int qtype, const Plan& pl, bool f32, bool unsplit, long long units, long long tiles, int grid, int n_sm) {
  if (pl.wt != 128 || (f32 && pl.nt > 128)) return false;
  if ((long long)grid * units >= 1LL << 32) return false;      // what first_group multiplies in 32 bits (no matrix that fits the GPU gets here: see there)
  if (unsplit) return true;
  if (grid > 8 * tiles) return false;
  return !f32 || pl.nt <= (qtype == B200Q_Q4_0 ? 48 : 32) || units >= (pl.nt <= 64 ? 4LL : 10LL) * n_sm;
}
template <int QT, bool F32>
int launch_tmem(StreamParams& p, int grid, cudaStream_t st) {
  auto kern = qgemm_tmem_kernel<QT, F32>;
  static PerDeviceFlag attr;
  const int dev = b200q_current_device();
  if (dev < 0) return B200Q_ERR_CUDA;
  if (!attr.test(dev)) {
    B200Q_CHECK_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, RING_BYTES));
    attr.set(dev);
  }
  // tensor memory: accumulators, then up to 4 slots of weights; shared memory: a K group of activations per slot, 2 to 6 stages of packed weights, and what is left
  // of a tile's accumulators once they have been read
  const int x_bytes = p.nt * (F32 ? 512 : 256), one = w_stage_bytes(QT), dump = p.nt * 512;
  p.d_cols = ceil_div(F32 && !p.unsplit ? 2 * p.nt : p.nt, 32) * 32;
  p.slots = std::min({MAX_T_SLOTS, (512 - p.d_cols) / A_COLS<F32>, (RING_BYTES - 2 * one) / x_bytes});
  p.dump = p.slots * x_bytes + 2 * one + dump <= RING_BYTES ? dump : 0;
  p.ahead = std::min(MAX_W_STAGES, (RING_BYTES - p.slots * x_bytes - p.dump) / one);
  const size_t smem = (size_t)p.slots * x_bytes + (size_t)p.ahead * one + p.dump;
  if (p.dump) p.dump = (int)smem - dump;
  B200Q_CHECK_CUDA(launch_k(kern, dim3(grid), dim3(T_THREADS), smem, st, true, p));
  return B200Q_OK;
}

}  // namespace

int b200q_qgemm_stream_status_take(int* status) {
  int zero = 0;
  B200Q_CHECK_CUDA(cudaMemcpyFromSymbol(status, g_tc_status, sizeof(int)));
  B200Q_CHECK_CUDA(cudaMemcpyToSymbol(g_tc_status, &zero, sizeof(int)));
  return B200Q_OK;
}

// CTAs of a launch: one per SM, but at least two K groups each (below that filling and draining the pipeline is all that a CTA does)
static int stream_grid(long long units, int n_sm) {
  const long long g = (units + 1) / 2, most = n_sm < (int)(COUNTER_BYTES / sizeof(unsigned)) ? n_sm : (int)(COUNTER_BYTES / sizeof(unsigned));
  return (int)(g < most ? g : most);
}

// the rows' scales, counters and partial sums behind the activation tiles; n_out = 0: enough for any
static size_t split_workspace(const Plan& pl, int n_out, int kgroups, int n_sm) {
  long long parts = 2LL * n_sm;
  if (n_out > 0) {
    const long long tiles = (long long)ceil_div(n_out, pl.wt) * pl.tok_tiles;
    const int grid = stream_grid(tiles * kgroups, n_sm);
    parts = tiles < grid ? grid + tiles : 2 * grid;
  }
  return scale_bytes(pl) + COUNTER_BYTES + (size_t)parts * pl.wt * pl.nt * sizeof(float);
}

// Room for the activation tiles: enough to run, tiles then going whole to the CTAs.  Equal tiles of up to 256 rows may hold more rows than m rounded up to 128
// (625 rows: 3 x 224), never fewer than a smaller m has.
extern "C" size_t b200q_qgemm_workspace_bytes(int m, int n_in) {
  if (m <= 0 || n_in <= 0) return 0;
  const Plan pl = make_plan(m, 0, 0);
  const size_t rows = std::max((size_t)ceil_div(m, 128) * 128, (size_t)pl.tok_tiles * pl.nt);
  return rows * ceil_div(n_in, GROUP_ELEMS) * GROUP_ELEMS * 4;
}
// ... with room for the rows' scales
extern "C" size_t b200q_qgemm_unsplit_workspace_bytes(int m, int n_in) {
  return m <= 0 || n_in <= 0 ? 0 : align256(b200q_qgemm_workspace_bytes(m, n_in)) + scale_bytes(make_plan(m, 0, 0));
}
extern "C" size_t b200q_qgemm_workspace_bytes_for(int m, int n_out, int n_in) {
  if (m <= 0 || n_in <= 0 || n_out < 0) return 0;
  const int n_sm = b200q_sm_count();
  return align256(b200q_qgemm_workspace_bytes(m, n_in)) + split_workspace(make_plan(m, n_out, n_sm > 0 ? n_sm : 148), n_out, ceil_div(n_in, GROUP_ELEMS), n_sm > 0 ? n_sm : 148);
}

// norm_weight (fp16 [n_in], fp32 activations only): the RMSNorm in front of the Linear, applied while the rows are split.
int b200q_qgemm_chain(int qtype, const void* w_packed, const void* x, int x_dtype, const void* norm_weight, float norm_eps, const void* bias_f16, const void* residual,
                      int epilogue, void* y, int y_dtype, int m, int n_out, int n_in, void* workspace, size_t workspace_bytes, cudaStream_t st, bool pdl, bool unsplit,
                      const b200q_row_input* row) {
  if (!w_packed || !x || !y || !workspace || m <= 0 || n_out <= 0 || n_in <= 0) return B200Q_ERR_BAD_ARG;
  if (epilogue != B200Q_EPI_LINEAR && epilogue != B200Q_EPI_SILU_MUL) return B200Q_ERR_BAD_ARG;
  if (epilogue == B200Q_EPI_SILU_MUL && (bias_f16 || residual || n_out % 16)) return B200Q_ERR_BAD_ARG;
  if (qtype == B200Q_Q6_K) return B200Q_ERR_UNSUPPORTED;
  if (qtype != B200Q_Q4_0 && qtype != B200Q_Q8_0) return B200Q_ERR_BAD_ARG;
  if ((x_dtype != B200Q_F32 && x_dtype != B200Q_F16) || (y_dtype != B200Q_F32 && y_dtype != B200Q_F16)) return B200Q_ERR_BAD_ARG;
  if (norm_weight && x_dtype != B200Q_F32) return B200Q_ERR_BAD_ARG;
  if (n_in % 32) return B200Q_ERR_BAD_SHAPE;
  if (((uintptr_t)w_packed | (uintptr_t)x | (uintptr_t)workspace | (uintptr_t)norm_weight) & 15) return B200Q_ERR_MISALIGNED;
  Plan pl = make_plan(m, 0, 0);                                // the activations' tiling does not depend on the device
  const bool f32 = x_dtype == B200Q_F32;
  const int kgroups = ceil_div(n_in, GROUP_ELEMS);
  const size_t xt_bytes = align256(tiles_bytes(pl, kgroups, f32));
  if (workspace_bytes < b200q_qgemm_workspace_bytes(m, n_in)) return B200Q_ERR_TOO_LARGE;
  const int n_sm = b200q_sm_count();
  if (n_sm <= 0) return B200Q_ERR_CUDA;
  pl = make_plan(m, n_out, n_sm);
  StreamParams p;
  p.w = (const uint8_t*)w_packed;
  p.xt = (const unsigned char*)workspace;
  p.down = f32 && workspace_bytes >= xt_bytes + scale_bytes(pl) ? (const float*)((unsigned char*)workspace + xt_bytes) : nullptr;
  p.counters = (unsigned*)((unsigned char*)workspace + xt_bytes + scale_bytes(pl));
  p.part = (float*)((unsigned char*)p.counters + COUNTER_BYTES);
  p.bias = (const __half*)bias_f16; p.residual = residual; p.y = y;
  p.m = m; p.n_out = n_out; p.kgroups = kgroups; p.n_row_tiles = ceil_div(n_out, TILE_ROWS);
  p.nt = pl.nt; p.tok_tiles = pl.tok_tiles;
  // Slots of unpacked weights and activations, 2 K groups or 3 (256 activation rows) to 5 steps; what they leave is for the packed blocks ahead:
  // at least two groups of Q4_0 (or one of Q8_0, whose blocks are twice as large) unless even two K groups leave less.
  const int slot = slot_bytes(pl, f32), one = ahead_bytes(qtype);
  p.slots = (RING_BYTES - (qtype == B200Q_Q4_0 ? 2 : 1) * one) / slot;
  if (p.slots > MAX_SLOTS) p.slots = MAX_SLOTS;
  p.ahead = (RING_BYTES - p.slots * slot) / one;
  if (p.ahead > MAX_AHEAD) p.ahead = MAX_AHEAD;
  p.y_f16 = y_dtype == B200Q_F16; p.silu_mul = epilogue == B200Q_EPI_SILU_MUL;
  p.tiles = ceil_div(n_out, pl.wt) * pl.tok_tiles;
  p.units = (long long)p.tiles * kgroups;
  const bool split = !unsplit && workspace_bytes >= xt_bytes + split_workspace(pl, n_out, kgroups, n_sm);
  p.grain = split ? 1 : kgroups; p.unsplit = !split;
  const int grid = split ? stream_grid(p.units, n_sm) : (p.tiles < n_sm ? p.tiles : n_sm);
  p.dump = p.d_cols = 0;
  // one CTA of the splitting kernel: 8 rows x the whole width, or a part of it where there are few rows (and, of fp32 rows, more than a CTA keeps in registers)
  const int row_groups = pl.tok_tiles * pl.nt / 8, n_chunks = kgroups * 16;
  const int parts = row_groups >= n_sm || (f32 && n_chunks <= SPLIT_HOLD * SPLIT_THREADS / 8) ? 1 : (row_groups * 4 >= n_sm || n_chunks < 256 ? 4 : 8);
  const int per = ceil_div(n_chunks, parts);
  const dim3 sgrid(row_groups, ceil_div(n_chunks, per));      // rows along x: y ends at 65535
  const bool cluster = f32 && sgrid.y > 1;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = sgrid; cfg.blockDim = dim3(SPLIT_THREADS); cfg.stream = st;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = pdl;
  attr[1].id = cudaLaunchAttributeClusterDimension;
  attr[1].val.clusterDim.x = 1; attr[1].val.clusterDim.y = sgrid.y; attr[1].val.clusterDim.z = 1;
  cfg.attrs = attr; cfg.numAttrs = cluster ? 2 : 1;
  const int n_counters = split ? grid : 0;
  if (row) {
    if (m != 1 || !f32 || split || n_in % 8 || norm_weight) return B200Q_ERR_BAD_ARG;
    if (n_in > B200Q_ROW_INPUT_MAX) return B200Q_ERR_TOO_LARGE;
    static PerDeviceFlag attr_set;
    const int dev = b200q_current_device();
    if (dev < 0) return B200Q_ERR_CUDA;
    if (!attr_set.test(dev)) {      // (without it, 48 KB with the static part)
      B200Q_CHECK_CUDA(cudaFuncSetAttribute(prepare_row_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, B200Q_ROW_INPUT_MAX * (int)sizeof(float)));
      attr_set.set(dev);
    }
    B200Q_CHECK_CUDA(launch_k(prepare_row_kernel, dim3(1), dim3(ROW_THREADS), (size_t)n_in * sizeof(float), st, pdl, *row, n_in, kgroups, pl.nt, (unsigned char*)p.xt,
                              (float*)p.down));
  } else if (f32)
    B200Q_CHECK_CUDA(cudaLaunchKernelEx(&cfg, cluster ? split_rows_kernel<float, true> : split_rows_kernel<float, false>, (const float*)x, (const __half*)norm_weight, norm_eps, m,
                                        n_in, kgroups, pl.nt, per, (unsigned char*)p.xt, p.counters, n_counters, (float*)p.down, unsplit ? 0.f : 1.f));
  else
    B200Q_CHECK_CUDA(cudaLaunchKernelEx(&cfg, split_rows_kernel<__half, false>, (const __half*)x, (const __half*)nullptr, 0.f, m, n_in, kgroups, pl.nt, per,
                                        (unsigned char*)p.xt, p.counters, n_counters, (float*)nullptr, 0.f));
  const bool tmem = takes_tmem(qtype, pl, f32, p.unsplit, p.units, p.tiles, grid, n_sm);
#define STREAM_CASE(QT) (tmem ? (f32 ? launch_tmem<QT, true>(p, grid, st) : launch_tmem<QT, false>(p, grid, st)) \
                         : pl.wt == 256 ? (f32 ? launch_stream<QT, 256, true>(p, grid, st) : launch_stream<QT, 256, false>(p, grid, st)) \
                                        : (f32 ? launch_stream<QT, 128, true>(p, grid, st) : launch_stream<QT, 128, false>(p, grid, st)))
  return qtype == B200Q_Q4_0 ? STREAM_CASE(B200Q_Q4_0) : STREAM_CASE(B200Q_Q8_0);
#undef STREAM_CASE
}

extern "C" int b200q_qgemm_ws_norm(int qtype, const void* w_packed, const void* x, int x_dtype, const void* norm_weight, float norm_eps,
                                   const void* bias_f16, const void* residual, int epilogue, void* y, int y_dtype, int m, int n_out, int n_in,
                                   void* workspace, size_t workspace_bytes, int unsplit, void* stream) {
  return b200q_qgemm_chain(qtype, w_packed, x, x_dtype, norm_weight, norm_eps, bias_f16, residual, epilogue, y, y_dtype, m, n_out, n_in, workspace,
                           workspace_bytes, (cudaStream_t)stream, false, unsplit != 0);
}
extern "C" int b200q_qgemm_ws(int qtype, const void* w_packed, const void* x, int x_dtype, const void* bias_f16, const void* residual, int epilogue,
                              void* y, int y_dtype, int m, int n_out, int n_in, void* workspace, size_t workspace_bytes, void* stream) {
  return b200q_qgemm_ws_norm(qtype, w_packed, x, x_dtype, nullptr, 0.f, bias_f16, residual, epilogue, y, y_dtype, m, n_out, n_in, workspace,
                             workspace_bytes, 0, stream);
}
