// The streaming GEMM for few activation rows (qgemm_stream.cu includes this; its parameters, unpacking and store_outputs are used here): unpacked weights reach the
// tensor core through tensor memory instead of shared memory.
//
// Why: with the weights (128 rows, the MMA's A operand) in shared memory an instruction takes 40 to 57 cycles up to N = 96, whatever its N; from tensor memory it takes
// 10 at N = 16, 25 at 48, 49 at 96, the time of its multiplications.  And nothing passes the proxy between a thread's stores and the tensor core any more.
//
// What paces it, and what follows from that:
//  * the thread that issues the MMAs: 4 unpack warps share its scheduler, so each of its instructions takes 7 to 8 cycles and the answer of a barrier that is ready
//    250.  A slot is a whole K group (24 instructions, one barrier for weights and activations), the next slot's barrier is asked before they are issued, and its loop is
//    kept short.  Slots of half a K group with two barriers: 1000 cycles a slot where the MMAs need 300, no faster than shared memory (8B gate / up, 45 rows: 74 us).
//  * the unpack warps: packed weights come as bulk copies of a row tile's K groups.  As one cp.async per lane a round's copies took 900 cycles (53 us).  They too ask
//    for their next barriers before they unpack.
//  * the end of a segment: the accumulators are read by all warps at once and are free again; a whole tile's outputs are computed from shared memory by four warps of
//    their own while the next tile goes on; the CTA that finishes a split tile last does not store its own part.
#pragma once

namespace {

constexpr int EPI_WARPS = 4;
constexpr int T_MMA = 0, T_COPY = 1, T_WCOPY = 2, T_SETUP = 3, T_UNPACK = 4, T_EPI = T_UNPACK + UNPACK_WARPS, T_THREADS = (T_EPI + EPI_WARPS) * 32;
// 8 unpack warps fill a slot, two such groups in turn.  Not more groups than slots: a group that is two uses of a slot ahead would take its barrier's phase for the one
// before.  Stages of two K groups at most: a group may fill one slot ahead of a segment's end, not two.
constexpr int MAX_T_SLOTS = 4, MAX_W_STAGES = 6;
template <bool F32> constexpr int A_COLS = F32 ? 128 : 64;      // tensor-memory columns of a slot's weights: a K group of high halves, then of remainders
// Packed weights wait in shared memory as they are: stages of 8 row tiles (128 rows) x W_GROUPS K groups, a bulk copy per row tile
constexpr int W_GROUPS = 2;
__host__ __device__ constexpr int w_stage_bytes(int qt) { return 8 * W_GROUPS * tile_bytes(qt); }

struct SharedT {
  uint64_t full[MAX_T_SLOTS], empty[MAX_T_SLOTS], w_full[MAX_W_STAGES], w_empty[MAX_W_STAGES], acc_full, acc_empty, dump_full, dump_free, early, stored[2], counted[2], drained;
  uint32_t tmem, last[2], others;
  int abort;
};
#define TBAR(sb, member) ((sb) + (uint32_t)offsetof(SharedT, member))

// Asks only: test_wait.  try_wait suspends the thread for a while if the answer is no, and some of these barriers are never completed (the slot after the last one).
__device__ __forceinline__ uint32_t bar_ready(uint32_t bar, uint32_t parity) {
  uint32_t ok;
  asm volatile("{\n.reg .pred p;\nmbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\nselp.u32 %0, 1, 0, p;\n}" : "=r"(ok) : "r"(bar), "r"(parity) : "memory");
  return ok;
}
// Bounded wait: false once another role has given up, or when the time is over (then the others are told).  Out of line: it is called in a dozen places.
__device__ __noinline__ bool t_wait_on(uint32_t sb, uint32_t bar, uint32_t parity) {
  for (int i = 0; i < (1 << 20); i++) {
    uint32_t ok, gone;
    asm volatile("{\n.reg .pred p;\nmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2, %3;\nselp.u32 %0, 1, 0, p;\n}"
                 : "=r"(ok) : "r"(bar), "r"(parity), "r"(2000) : "memory");
    if (ok) return true;
    asm volatile("ld.volatile.shared::cta.u32 %0, [%1];" : "=r"(gone) : "r"(TBAR(sb, abort)) : "memory");
    if (gone) return false;
  }
  asm volatile("st.volatile.shared::cta.u32 [%0], 1;" ::"r"(TBAR(sb, abort)) : "memory");
  atomicExch(&g_tc_status, 1);
  return false;
}
__device__ __forceinline__ bool t_wait(uint32_t sb, uint32_t bar, uint32_t parity) { return bar_ready(bar, parity) || t_wait_on(sb, bar, parity); }
__device__ __forceinline__ void mma_ts(uint32_t d, uint32_t a, uint32_t b_lo, uint32_t hi, uint32_t idesc, uint32_t acc) {
  asm volatile("{\n.reg .pred p;\n.reg .b64 b;\nmov.b64 b, {%2, %3};\nsetp.ne.u32 p, %5, 0;\n"
               "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], b, %4, p;\n}"
               ::"r"(d), "r"(a), "r"(b_lo), "r"(hi), "r"(idesc), "r"(acc) : "memory");
}
__device__ __forceinline__ void st_tmem16(uint32_t a, const uint4 (&v)[4]) {
  asm volatile("tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16};"
               ::"r"(a), "r"(v[0].x), "r"(v[0].y), "r"(v[0].z), "r"(v[0].w), "r"(v[1].x), "r"(v[1].y), "r"(v[1].z), "r"(v[1].w),
                 "r"(v[2].x), "r"(v[2].y), "r"(v[2].z), "r"(v[2].w), "r"(v[3].x), "r"(v[3].y), "r"(v[3].z), "r"(v[3].w) : "memory");
}
__device__ __forceinline__ uint4 ld_shared4(uint32_t addr) {
  uint4 v;
  asm volatile("ld.shared.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(addr) : "memory");
  return v;
}

// Accumulator columns (activation rows) a thread takes at a time at the end of a segment: 8 of half-precision rows (4608 x 3584, 301 rows: 31.9 us with 4, 28.3), but the
// fp32 kernels have no registers for that (spills in the unpack loop: 4096 x 4096, 45 rows 22.2 us, 24.3 with 8).
template <bool F32> constexpr int N_COLS = F32 ? 4 : 8;
__device__ __forceinline__ void ld_columns(uint32_t a, uint32_t (&v)[4]) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x4.b32 {%0,%1,%2,%3}, [%4];" : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]) : "r"(a));
}
__device__ __forceinline__ void ld_columns(uint32_t a, uint32_t (&v)[8]) { ld_tmem(a, v); }

struct Segment { int seg, tile, k0, k1; bool last; };      // number within the CTA's, K groups k0 .. k1 of tile; `last`: the CTA's last
// The deal in 32 bits: K groups of all tiles times CTAs are below 2^32 (takes_tmem asks).  A matrix that fits the GPU has that: 3.2e11 4-bit weights are 2e7 K groups of
// 128 rows, and more than one tile of activation rows meets tiles of 128 weight rows only where those are few (make_plan).
__device__ __forceinline__ uint32_t first_group(uint32_t c, const StreamParams& p, uint32_t g) { return p.grain == 1 ? c * (uint32_t)p.units / g : c * p.tiles / g * p.grain; }
__device__ __forceinline__ int cta_of_group(uint32_t unit, const StreamParams& p, uint32_t g) { return (int)(((unit + 1) * g - 1) / (uint32_t)p.units); }
// the first of the CTAs that have a tile, and how many
__device__ __forceinline__ int2 tile_ctas(const StreamParams& p, int tile) {
  const int c0 = cta_of_group((uint32_t)tile * p.kgroups, p, gridDim.x);
  return make_int2(c0, cta_of_group((uint32_t)(tile + 1) * p.kgroups - 1, p, gridDim.x) - c0 + 1);
}

// What all 20 warps do at the end of a segment: warp q of the five of a row quarter reads every fifth group of NC accumulator columns.  A whole tile's go to shared
// memory (`dump`, where there is room; the epilogue warps alone make outputs of them, the others go on with the next segment), to a partial sum, or become outputs at once.
// One loop for all of it: this code runs once or twice a launch, and what it takes is mostly the time to fetch its instructions (with store_outputs in
// six places 4096 x 4096 took 38 us).
template <bool F32>
__device__ __forceinline__ bool finish_segment_t(const StreamParams& p, SharedT& sh, uint32_t sb, const Segment& g, int first_tile, bool first_part, int& dumps, uint32_t dump) {
  constexpr int PARTS = (UNPACK_WARPS + EPI_WARPS) / 4, NC = N_COLS<F32>;
  const int tid = threadIdx.x, lane = tid & 31, sub = (tid >> 5) & 3, part = (tid >> 7) - T_UNPACK / 4;
  const int row = sub * 32 + lane;
  int tile = g.tile;
  const bool whole = g.k0 == 0 && g.k1 == p.kgroups, epi = tid >= T_EPI * 32, asks = tid == T_EPI * 32;
  const int c = blockIdx.x, groups = p.nt / NC, second = F32 && !p.unsplit ? p.nt : 0;
  int2 ctas = make_int2(c, 1);
  if (!whole) ctas = tile_ctas(p, g.tile);
  const size_t slot = (size_t)128 * p.nt;
  const bool partial_last = !whole && g.last, dumped = whole && !g.last && dump;
  // The last to finish a tile need not store its own part: are all the others there already?
  if (partial_last && asks) {
    unsigned there;
    asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(there) : "l"(p.counters + ctas.x) : "memory");
    const bool others = there == (unsigned)ctas.y - 1;
    if (others) p.counters[ctas.x] = 0;
    sh.others = others;
    bar_arrive(TBAR(sb, early));
  }
  bool ok = t_wait(sb, TBAR(sb, acc_full), g.seg & 1) && (!partial_last || t_wait(sb, TBAR(sb, early), 0));
  if (dumped) ok = ok && t_wait(sb, TBAR(sb, dump_free), (dumps & 1) ^ 1);
  if (!__all_sync(0xffffffffu, ok)) return false;
  const bool alone = partial_last && *reinterpret_cast<volatile uint32_t*>(&sh.others);
  const bool kept = !whole && !alone;          // as a partial sum
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t ta = sh.tmem + ((uint32_t)(sub * 32) << 16), mine_s = dump + row * 16;
  float* const parts = p.part + row * 4;       // [group of 4 columns][row][4]: a warp's store is 512 contiguous bytes
  float* const mine = parts + part_slot(p, c, tile, c == ctas.x) * slot;
  int cg = part, step = PARTS;
  bool from_dump = false;
#pragma unroll 1
  for (int pass = 0; pass < 3; pass++) {       // from the accumulators, from where they were left, and at the CTA's end its first segment's tile
    const int ft = p.tok_tiles == 1 ? tile : tile / p.tok_tiles, tt = tile - ft * p.tok_tiles, feat = ft * 128 + row;
#pragma unroll 1
    for (; cg < groups; cg += step) {
      float v[NC] = {};
      int own = -1, n_add = 0;
      if (pass == 0) {
        uint32_t a[NC], b[NC];
        ld_columns(ta + cg * NC, a);
        if (second) ld_columns(ta + second + cg * NC, b);
        asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
        for (int j = 0; j < NC; j++) v[j] = second ? __uint_as_float(a[j]) + __uint_as_float(b[j]) : __uint_as_float(a[j]);
        if (dumped || kept) {
#pragma unroll
          for (int j = 0; j < NC; j += 4) {
            const uint4 f = make_uint4(__float_as_uint(v[j]), __float_as_uint(v[j + 1]), __float_as_uint(v[j + 2]), __float_as_uint(v[j + 3]));
            if (dumped) st_shared(mine_s + (cg * NC + j) * 512, f);
            else __stcg(reinterpret_cast<uint4*>(mine + (size_t)(cg * NC + j) * 128), f);
          }
          continue;
        }
        if (alone) { own = c - ctas.x; n_add = ctas.y; }
      } else if (from_dump) {
#pragma unroll
        for (int j = 0; j < NC; j += 4) {
          const uint4 f = ld_shared4(mine_s + (cg * NC + j) * 512);
          v[j] = __uint_as_float(f.x); v[j + 1] = __uint_as_float(f.y); v[j + 2] = __uint_as_float(f.z); v[j + 3] = __uint_as_float(f.w);
        }
      } else n_add = ctas.y;
      if (n_add) {                             // the parts in the order of K
        float w[NC] = {};
#pragma unroll(F32 ? 4 : 2)
        for (int s = 0; s < n_add; s++) {
#pragma unroll
          for (int j = 0; j < NC; j += 4) {
            const float4 f = __ldcg(reinterpret_cast<const float4*>(parts + part_slot(p, ctas.x + s, tile, s == 0) * slot + (size_t)(cg * NC + j) * 128));
            const bool mine = s == own;        // (loaded all the same: loads under a branch went one by one, 400 x 4096, 120 half-precision rows 41 us)
            w[j] += mine ? v[j] : f.x; w[j + 1] += mine ? v[j + 1] : f.y; w[j + 2] += mine ? v[j + 2] : f.z; w[j + 3] += mine ? v[j + 3] : f.w;
          }
        }
#pragma unroll
        for (int j = 0; j < NC; j++) v[j] = w[j];
      }
      store_outputs(p, v, feat, tt * p.nt + cg * NC, lane);
    }
    cg = groups;
    if (pass == 0) {
      asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
      __syncwarp();
      if (lane == 0) {
        bar_arrive(TBAR(sb, acc_empty));
        if (dumped) bar_arrive(TBAR(sb, dump_full));
        if (kept) bar_arrive(TBAR(sb, stored) + 8 * g.last);
      }
      if (dumped) {
        dumps++;
        if (!epi) return true;
        if (!__all_sync(0xffffffffu, t_wait(sb, TBAR(sb, dump_full), (dumps & 1) ^ 1))) return false;
        from_dump = true;
        cg = 0; step = 1;                      // the epilogue warps alone
        continue;
      }
      // a CTA has at most two partial segments, its first and its last: a barrier pair each.  One thread's count releases what all have stored before the barrier
      // (a fence in every thread took 1900 cycles, under which the accumulators were not free).
      if (kept && asks && t_wait(sb, TBAR(sb, stored) + 8 * g.last, 0)) {
        unsigned old;
        asm volatile("atom.add.acq_rel.gpu.global.u32 %0, [%1], 1;" : "=r"(old) : "l"(p.counters + ctas.x) : "memory");
        const bool adds = old == (unsigned)ctas.y - 1;
        if (adds) p.counters[ctas.x] = 0;
        sh.last[g.last] = adds;
        bar_arrive(TBAR(sb, counted) + 8 * g.last);
      }
      if (!g.last) return true;
      if (kept) {
        if (!__all_sync(0xffffffffu, t_wait(sb, TBAR(sb, counted) + 8, 0))) return false;
        if (*reinterpret_cast<volatile uint32_t*>(&sh.last[1])) cg = part;
      }
    } else if (pass == 1) {
      if (from_dump) {
        __syncwarp();
        if (lane == 0) bar_arrive(TBAR(sb, dump_free));
        return true;
      }
      // If this CTA was the last at the tile its first segment is a part of, the parts are added now, by all warps (by four of them in between: 15 us at
      // 4096 x 4096, where the CTA has nothing else left to do)
      if (!first_part) break;
      if (!__all_sync(0xffffffffu, t_wait(sb, TBAR(sb, counted), 0))) return false;
      if (!*reinterpret_cast<volatile uint32_t*>(&sh.last[0])) break;
      tile = first_tile;
      ctas = tile_ctas(p, tile);
      cg = part;
    }
  }
  return true;
}

template <int QT, bool F32>
__global__ void __launch_bounds__(T_THREADS, 1) qgemm_tmem_kernel(const StreamParams p) {
  constexpr int TB = tile_bytes(QT), W_STAGE = w_stage_bytes(QT), W_ROWS = W_GROUPS * TB, AC = A_COLS<F32>;
  extern __shared__ __align__(128) unsigned char dyn[];
  __shared__ SharedT sh;
  const uint32_t sb = pinned(s32(&sh)), ring = pinned(s32(dyn));
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int G = gridDim.x, c = blockIdx.x;
  // the CTA's K groups: n_units from group k_first of tile tile_first on
  const uint32_t u0 = first_group(c, p, G);
  const int n_units = (int)(first_group(c + 1, p, G) - u0), tile_first = (int)(u0 / (uint32_t)p.kgroups), k_first = (int)(u0 - (uint32_t)tile_first * p.kgroups);
  const int nt = p.nt, x_rows = F32 ? 2 * nt : nt;
  const uint32_t x_step = (uint32_t)x_rows * 64, x_bytes = 4 * x_step;      // activations of 32 columns and of a K group
  if (warp == T_SETUP) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], 512;" ::"r"(s32(&sh.tmem)) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  if (tid == T_UNPACK * 32) {
    // a slot is full when its 8 unpack warps and the copy thread have arrived and the copy's bytes are there; one commit empties it
    for (int i = 0; i < MAX_T_SLOTS; i++) { bar_init(TBAR(sb, full) + 8 * i, 9); bar_init(TBAR(sb, empty) + 8 * i, 1); }
    for (int i = 0; i < MAX_W_STAGES; i++) { bar_init(TBAR(sb, w_full) + 8 * i, 1); bar_init(TBAR(sb, w_empty) + 8 * i, UNPACK_WARPS); }
    bar_init(TBAR(sb, acc_full), 1); bar_init(TBAR(sb, acc_empty), EPI_WARPS + UNPACK_WARPS); bar_init(TBAR(sb, drained), 1);
    bar_init(TBAR(sb, dump_full), EPI_WARPS + UNPACK_WARPS); bar_init(TBAR(sb, dump_free), EPI_WARPS); bar_init(TBAR(sb, early), 1);
    bar_init(TBAR(sb, stored), EPI_WARPS + UNPACK_WARPS); bar_init(TBAR(sb, stored) + 8, EPI_WARPS + UNPACK_WARPS);
    bar_init(TBAR(sb, counted), 1); bar_init(TBAR(sb, counted) + 8, 1);
    sh.abort = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  pdl_launch_dependents();
  const uint32_t a_base = sh.tmem + p.d_cols, w_ring = ring + p.slots * x_bytes;
  auto open_segment = [&](int u, int seg, int& tile, int& k0, int& k1) {      // the one that starts at K group u of the CTA's
    tile = tile_first + seg; k0 = seg ? 0 : k_first; k1 = min(p.kgroups, k0 + n_units - u);
  };

  if (warp == T_COPY) {
    if (elect_one()) {
      pdl_wait();                                        // the activation tiles are the previous kernel's (generic stores, read by bulk copies here)
      asm volatile("fence.proxy.async.global;" ::: "memory");
      bool ok = true;
      int n = 0, slot = 0;
      uint32_t par = 1;
      for (int u = 0, seg = 0; u < n_units && ok; seg++) {
        int tile, k0, k1;
        open_segment(u, seg, tile, k0, k1);
        const unsigned char* src = p.xt + ((size_t)(tile % p.tok_tiles) * p.kgroups + k0) * x_bytes;
        for (int s = k1 - k0; s > 0; s--, n++, src += x_bytes) {
          if (!t_wait(sb, TBAR(sb, empty) + 8 * slot, par)) { ok = false; break; }
          const uint32_t dst = ring + slot * x_bytes, bar = TBAR(sb, full) + 8 * slot;
          asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(x_bytes) : "memory");
          for (uint32_t o = 0; o < x_bytes; o += 16384)
            asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
                         ::"r"(dst + o), "l"(src + o), "r"(min(16384u, x_bytes - o)), "r"(bar) : "memory");
          if (++slot == p.slots) { slot = 0; par ^= 1; }
        }
        u += k1 - k0;
      }
      // Nothing may still be landing in shared memory when the CTA leaves.  After a failed wait a slot's unpack warps may never arrive, so its
      // barrier cannot tell; the copies are done long before the time that wait took, and one more is spent here.
      for (int j = max(0, n - p.slots); j < n; j++)
        if (!wait_bar(TBAR(sb, full) + 8 * (j % p.slots), (j / p.slots) & 1)) break;
    }
  } else if (warp == T_WCOPY) {
    if (elect_one()) {                                   // weights do not depend on earlier kernels: no waiting for them
      bool ok = true;
      int n = 0, st = 0;
      uint32_t par = 1;
      for (int u = 0, seg = 0; u < n_units && ok; seg++) {
        int tile, k0, k1;
        open_segment(u, seg, tile, k0, k1);
        u += k1 - k0;
        const int rt = tile / p.tok_tiles * 8, rows = min(8, p.n_row_tiles - rt);      // past the last row tile: whatever is there, for rows nobody reads
        const uint8_t* src = p.w + ((size_t)rt * p.kgroups + k0) * TB;
        const size_t next_rows = (size_t)p.kgroups * TB;
        for (int k = k0; k < k1; k += W_GROUPS, n++, src += W_ROWS) {
          if (!t_wait(sb, TBAR(sb, w_empty) + 8 * st, par)) { ok = false; break; }
          const uint32_t bytes = (uint32_t)min(W_GROUPS, k1 - k) * TB, bar = TBAR(sb, w_full) + 8 * st;
          uint32_t dst = w_ring + st * W_STAGE;
          asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes * rows) : "memory");
          const uint8_t* s = src;
#pragma unroll 1
          for (int i = 0; i < rows; i++, dst += W_ROWS, s += next_rows)
            asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(dst), "l"(s), "r"(bytes), "r"(bar) : "memory");
          if (++st == p.ahead) { st = 0; par ^= 1; }
        }
      }
      for (int j = max(0, n - p.ahead); j < n; j++)
        if (!wait_bar(TBAR(sb, w_full) + 8 * (j % p.ahead), (j / p.ahead) & 1)) break;
    }
  } else if (warp == T_MMA) {
    // Shuffled, a value is known to be the same for the warp and can stay where the tensor core's operands have to be.
    const uint32_t d = __shfl_sync(0xffffffffu, sh.tmem, 0), a0 = __shfl_sync(0xffffffffu, a_base, 0);
    const uint32_t x0 = __shfl_sync(0xffffffffu, (ring >> 4) | ((uint32_t)x_rows << 16), 0), full0 = __shfl_sync(0xffffffffu, TBAR(sb, full), 0);
    if (elect_one()) {
      bool ok = true;
      const bool two_sums = F32 && !p.unsplit;
      // Every instruction has the one shape 128 x nt, and what two of them add to is the same columns: in that order they are added.  (wh x [xh | xl] as one instruction
      // of 2 nt columns and wl xh in half of its columns were two shapes in one accumulator, between which no order is promised.)
      const uint32_t id = make_idesc(128, nt);
      // Two sums: the remainders' products are all added up beside the high parts', where the tensor core's truncating additions to a small sum lose little: one
      // addition to the large sum per 16 columns instead of three (28672 x 4096, 45 rows: 7.3e-6 of the result with two, 4.0e-6 so).
      const uint32_t d_lo = two_sums ? d + nt : d;
      const uint32_t desc_hi = (uint32_t)(make_desc(0, 0, 128) >> 32), x_next = x_bytes >> 4, k32 = x_step >> 4, k16 = 2 * x_rows;
      constexpr uint32_t TO_EMPTY = offsetof(SharedT, empty) - offsetof(SharedT, full);
      int seg = 0, left = p.slots;                            // slots until the ring starts again
      uint32_t par = 0, ready = 0, a = a0, x = x0, full = full0;
      for (int u = 0; u < n_units && ok; seg++) {
        int tile, k0, k1;
        open_segment(u, seg, tile, k0, k1);
        u += k1 - k0;
        if (!t_wait(sb, TBAR(sb, acc_empty), (seg & 1) ^ 1)) { ok = false; break; }
        uint32_t acc = 0, acc_lo = two_sums ? 0 : 1;
#pragma unroll 1
        for (int s = k1 - k0; s > 0; s--) {
          if (!ready && !t_wait(sb, full, par)) { ok = false; break; }
          asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
          const uint32_t wa = a, xa = x, bar = full + TO_EMPTY;
          a += AC; x += x_next; full += 8;
          if (--left == 0) { left = p.slots; a = a0; x = x0; full = full0; par ^= 1; }
          ready = bar_ready(full, par);      // the next slot's: the answer comes back while this slot's instructions are issued
#pragma unroll
          for (int kk = 0; kk < 8; kk++) {
            const uint32_t xh = xa + (kk >> 1) * k32 + (kk & 1) * k16;
            mma_ts(d, wa + kk * 8, xh, desc_hi, id, kk ? 1u : acc);
            if (F32) {
              mma_ts(d_lo, wa + kk * 8, xh + nt, desc_hi, id, kk ? 1u : acc_lo);
              mma_ts(d_lo, wa + 64 + kk * 8, xh, desc_hi, id, 1u);
            }
          }
          acc = acc_lo = 1;
          commit(bar);
        }
        if (ok) commit(TBAR(sb, acc_full));
      }
      commit(TBAR(sb, drained));                              // also on the way out after a failed wait: MMAs issued must be done before tensor memory goes back
      wait_bar(TBAR(sb, drained), 0);
    }
  } else if (warp >= T_UNPACK) {
    bool ok = true;
    int dumps = 0;
    const uint32_t dump = p.dump ? ring + p.dump : 0;
    {
      // ------------------------------ unpack; the epilogue warps only finish segments ------------------------------
      // Lane quarter `qr` of the 128 rows; thread groups 0, 1 fill the even slots, 2, 3 the odd ones, each one half of a K group.  A thread takes two blocks.
      const bool epi = warp >= T_EPI;
      const int qr = warp & 3, turn = (warp - T_UNPACK) >> 3, pair = ((warp - T_UNPACK) >> 2) & 1;
      int slot = turn, n = 0, st = 0;
      uint32_t par = 1, w_par = 0;
      const uint32_t a_mine = a_base + ((uint32_t)(qr * 32) << 16) + pair * 32;
      // This lane's row (of the warp's two row tiles) in a stage.  The row's blocks are 64 bytes from the next row's: lanes 2, 3, 6, 7 .. read the second block
      // first, so that 8 lanes meet two to a bank instead of four.
      const int r = lane & 15;
      const bool swap = lane & 2;
      const uint32_t w_row = w_ring + (qr * 2 + (lane >> 4)) * W_ROWS;
      const uint32_t w_at = w_row + ((r >> 3) * (QT == B200Q_Q4_0 ? 32 : 64) + (r & 7) * 4 + pair * 2) * 16 + (swap ? 16 : 0);
      const uint32_t w_other = swap ? (uint32_t)-16 : 16u, w_scale = w_row + TB - 128 + (2 * (r & 7) + pair) * 8 + (r >> 3) * 4;
      // A segment is finished after this group's first slot of the next one: it gives the tensor core something to do meanwhile (two slots in all, no more than the ring has).
      Segment cur = {0, 0, 0, 0, false}, done = cur;
      bool pending = false;
      int u = 0;
      uint32_t slot_ready = 0, w_ready = 0;
      auto open = [&]() { open_segment(u, cur.seg, cur.tile, cur.k0, cur.k1); cur.last = u + (cur.k1 - cur.k0) >= n_units; };
      open();
      int k = cur.k0;
      while (ok) {
        const bool more = u < n_units;
        bool lead = !more || epi, seg_end = epi;
        if (more && !epi) {
          const int cnt = min(W_GROUPS, cur.k1 - k);
          if (!__all_sync(0xffffffffu, w_ready)) ok = __all_sync(0xffffffffu, t_wait(sb, TBAR(sb, w_full) + 8 * st, w_par));
          if (!ok) break;
          w_ready = 0;
          const uint32_t stage = st * W_STAGE, w_done = TBAR(sb, w_empty) + 8 * st;
          if (++st == p.ahead) { st = 0; w_par ^= 1; }
#pragma unroll 1
          for (int i = (turn ^ n) & 1; i < cnt; i += 2) {
            const uint32_t at = w_at + stage + i * TB;
            uint4 raw[2], rawb[2];
            raw[0] = ld_shared4(at); raw[1] = ld_shared4(at + w_other);
            if constexpr (QT == B200Q_Q8_0) { rawb[0] = ld_shared4(at + 512); rawb[1] = ld_shared4(at + 512 + w_other); }
            uint32_t d;
            asm volatile("ld.shared.u32 %0, [%1];" : "=r"(d) : "r"(w_scale + stage + i * TB) : "memory");
            if (!__all_sync(0xffffffffu, slot_ready)) ok = __all_sync(0xffffffffu, t_wait(sb, TBAR(sb, empty) + 8 * slot, par));
            if (!ok) break;
            w_ready = bar_ready(TBAR(sb, w_full) + 8 * st, w_par);      // the answers come back while the weights are unpacked
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            const uint32_t to = a_mine + slot * AC;
#pragma unroll
            for (int b = 0; b < 2; b++) {
              auto pick = [&](const uint4 (&q)[2]) {
                return make_uint4(swap ? q[1 - b].x : q[b].x, swap ? q[1 - b].y : q[b].y, swap ? q[1 - b].z : q[b].z, swap ? q[1 - b].w : q[b].w);
              };
              const uint4 qa = pick(raw);
              const uint32_t d2 = prmt(d, d, b ? 0x3232u : 0x1010u);
              uint4 hi[4], lo[4];
              if constexpr (QT == B200Q_Q4_0) {
                uint32_t v[4][4];
                q4_word(qa.x, v[0]); q4_word(qa.y, v[1]); q4_word(qa.z, v[2]); q4_word(qa.w, v[3]);
#pragma unroll
                for (int j = 0; j < 4; j++) {
                  const int x = (j & 1) * 2, y = (j >> 1) * 2;      // chunk j: words x, x + 1; low or high nibbles
                  const uint32_t r4[4] = {v[x][y], v[x][y + 1], v[x + 1][y], v[x + 1][y + 1]};
                  hi[j] = hi_lo(r4, d2, lo[j]);
                }
              } else {
                const uint4 qb = pick(rawb);
                hi[0] = q8_core(qa.x, qa.y, d2, lo[0]); hi[1] = q8_core(qa.z, qa.w, d2, lo[1]);
                hi[2] = q8_core(qb.x, qb.y, d2, lo[2]); hi[3] = q8_core(qb.z, qb.w, d2, lo[3]);
              }
              st_tmem16(to + b * 16, hi);
              if (F32) st_tmem16(to + 64 + b * 16, lo);
            }
            asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
            asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
            __syncwarp();
            if (lane == 0) bar_arrive(TBAR(sb, full) + 8 * slot);
            slot += 2;
            if (slot >= p.slots) { slot -= p.slots; par ^= 1; }
            slot_ready = bar_ready(TBAR(sb, empty) + 8 * slot, par);
            lead = true;
          }
          __syncwarp();
          if (!ok) break;
          if (lane == 0) bar_arrive(w_done);
          n += cnt;
          k += W_GROUPS;
          seg_end = k >= cur.k1;
        }
        if (pending && (lead || seg_end)) {
          if (done.seg == 0) pdl_wait();                   // the epilogue reads and writes what earlier kernels touched
          ok = __all_sync(0xffffffffu, finish_segment_t<F32>(p, sh, sb, done, tile_first, k_first != 0 && done.seg, dumps, dump));
          pending = false;
        }
        if (!more) break;
        if (seg_end) {
          done = cur; pending = true;
          u += cur.k1 - cur.k0;
          cur.seg++;
          if (u < n_units) { open(); k = cur.k0; }
        }
      }
    }
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (warp == T_SETUP) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, 512;" ::"r"(sh.tmem) : "memory");
}

}  // namespace
