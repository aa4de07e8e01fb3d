// Shared declarations for the sm_100a kernels and their C-ABI launchers.
#pragma once
#include <cuda_runtime.h>
#include <cuda_fp16.h>
#include <stdint.h>
#include <atomic>
#include "../../include/b200q.h"

#define B200Q_CHECK_CUDA(expr)                                   \
  do {                                                           \
    cudaError_t _e = (expr);                                     \
    if (_e != cudaSuccess) { b200q_set_cuda_error(_e); return B200Q_ERR_CUDA; } \
  } while (0)

void b200q_set_cuda_error(cudaError_t e);

// ---- launch chains.  Exported entry points launch their first kernel fully ordered behind whatever the caller has put on the stream; the `pdl`
// argument of the internal forms below is for calls whose predecessor on the stream is known to be a kernel of this library.
// one row of a GEMM that is not split, with what is in front of it: x += the weighted sum of the k rows dest_row of y (bf16; NULL: nothing), RMSNorm (norm_w NULL: none)
constexpr int B200Q_ROW_INPUT_MAX = 12288;      // values of such a row: it stands in shared memory (48 KB)
struct b200q_row_input { float* x; const void* y; const int32_t* dest_row; const float* weights; int k; const void* norm_w; float eps; };
int b200q_qgemm_chain(int qtype, const void* w_packed, const void* x, int x_dtype, const void* norm_weight, float norm_eps, const void* bias_f16, const void* residual,
                      int epilogue, void* y, int y_dtype, int m, int n_out, int n_in, void* workspace, size_t workspace_bytes, cudaStream_t st, bool pdl,
                      bool unsplit = false, const b200q_row_input* one = nullptr);
// out NULL: RoPE and the cache rows only
int b200q_attn_rows_chain(const float* qkv, void* k_cache, void* v_cache, int kv_dtype, const float* rope, int start_pos, int n_rows, int n_seqs, int n_heads,
                          int n_kv_heads, int head_dim, int rope_dim, int max_context, void* q_scratch, void* out, int out_dtype, cudaStream_t st, bool pdl);

// ---- per-device launcher state ---------------------------------------------------------
// One host process may drive several GPUs (tinygrad does: one process, one context per device,
// tinygrad/runtime/ops_cuda.py:97-134), and cudaFuncSetAttribute / the SM count belong to the device that is current.
// Launchers therefore keep what they cache in tables indexed by the current device.  Setting an attribute twice is
// harmless, so a relaxed atomic flag per device is all the thread safety the tables need.
constexpr int B200Q_MAX_DEVICES = 64;
struct PerDeviceFlag {
  std::atomic<int> v[B200Q_MAX_DEVICES];
  bool test(int dev) const { return v[dev].load(std::memory_order_acquire) != 0; }
  void set(int dev) { v[dev].store(1, std::memory_order_release); }
};
// reads and clears the status word of the decode-step kernels (decode.cu); folded into b200q_status_read_clear
// gives the result pool's unused blocks of a device back (pool.cu); false: there were none
bool b200q_pool_release(int dev);
// fp8 product with factors, bias and output type in the epilogue (mxfp8_gemm.cu)
int b200q_mx_gemm_scaled(const void* a_q, const void* b_q, const int32_t* off, int m_total, int n, int k, void* y, int y_dtype, int rows,
                         const float* fw, const float* fx, const float* bias, cudaStream_t st);
int b200q_mx_gemm_chain(const void* a_q, const void* a_e8, const void* b_q, const void* b_e8, const int32_t* off, const int32_t* ends, int n_experts, int m_total, int n,
                        int k, void* c_bf16, void* act_q, void* act_e8, int n_tokens, int topk, cudaStream_t st);
int b200q_moe_layer_chain(const b200q_moe_args* m, const void* x_bf16, const float* logits, int n_tokens, float* add_to, cudaStream_t st, bool pdl);
// out (fp32) and out_bf16 (either may be NULL): RMSNorm(x) * weight (prefill.cu)
int b200q_rmsnorm_rows_chain(const float* x, const void* weight_f16, float eps, int n_rows, int dim, float* out, void* out_bf16, cudaStream_t st);
int b200q_add_rows_gated_chain(float* x, const float* y, const float* gate_logit, int n_rows, int dim, cudaStream_t st);
int b200q_attn_rows_pos_chain(const float* qkv, void* k_cache, void* v_cache, int kv_dtype, const float* rope, const int32_t* pos_dev, int n_heads, int n_kv_heads, int head_dim,
                              int rope_dim, int max_context, void* q_scratch, void* out, int out_dtype, cudaStream_t st);
// one row times a packed matrix in fp32 (row_gemv.cu)
int b200q_row_gemv_chain(int qtype, const void* w_packed, const float* x, const void* norm_weight, float norm_eps, const void* bias_f16, const float* residual, int epilogue,
                         float* y, int n_out, int n_in, cudaStream_t st, bool pdl);
// behind the expert GEMMs: the weighted sums, added to add_to (mxfp8.cu)
int b200q_moe_combine_chain(const b200q_moe_args* m, int n_tokens, float* add_to, cudaStream_t st);
int b200q_moe_gemms_chain(const b200q_moe_args* m, int n_tokens, cudaStream_t st);
// one token: RMSNorm, router, choice and tables, quantised rows (moe_step.cu); xn (may be NULL): the normed row
bool b200q_moe_router_one_takes(const b200q_moe_args* m, int router_dtype);
int b200q_moe_router_one(const b200q_moe_args* m, const void* router, int router_dtype, const float* x, const void* norm_weight, float eps, float* xn, cudaStream_t st);
int b200q_decode_status_take(int* status);
int b200q_decode_step_status_take(int* status);   // the same for the whole-step kernel (decode_step.cu)
int b200q_peer_status_take(int* status);          // the same for the peer-memory collectives (peer.cu)
int b200q_qgemm_stream_status_take(int* status);  // the same for the many-row GEMM (qgemm_stream.cu)
int b200q_ep_status_take(int* status);            // the same for the expert-parallel exchange (ep.cu)
// current device index, or -1 (with the CUDA error recorded) if it cannot be had or is past the tables
int b200q_current_device();
// SM count of the current device (cached per device); 0 on error
int b200q_sm_count();

// ---- packed weight layout (see include/b200q.h for the byte-level description)
constexpr int TILE_ROWS = 16;       // output rows per tile (one mma.m16n8k16 A operand)
constexpr int GROUP_ELEMS = 128;    // K elements per tile: 4 quant blocks of 32 (Q4_0/Q8_0), half a super-block (Q6_K)

__host__ __device__ constexpr int tile_bytes(int qtype) {
  return qtype == B200Q_Q4_0 ? 1152 : qtype == B200Q_Q8_0 ? 2176 : qtype == B200Q_Q6_K || qtype == B200Q_Q6_K_WIDE ? 1696 : qtype == B200Q_Q4_K_WIDE ? 1216 : 0;
}

static inline int ceil_div(int a, int b) { return (a + b - 1) / b; }

// ---- programmatic dependent launch (PDL).  Every kernel calls pdl_wait() before it
// touches memory another kernel wrote, so a chain of launches stays ordered.
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void pdl_launch_dependents() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

// Launch with the programmatic-stream-serialization attribute when `pdl` is set.
template <typename... KArgs, typename... Args>
static inline cudaError_t launch_k(void (*kernel)(KArgs...), dim3 grid, dim3 block, size_t smem, cudaStream_t stream, bool pdl,
                                   Args... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid; cfg.blockDim = block; cfg.dynamicSmemBytes = smem; cfg.stream = stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr; cfg.numAttrs = pdl ? 1 : 0;
  return cudaLaunchKernelEx(&cfg, kernel, KArgs(args)...);
}

// ---- mailboxes in peer memory ---------------------------------------------------------------------------------------
// A mailbox word is 32 bits: the fp32 value, or MAILBOX_EMPTY.  One aligned 32-bit store / load is atomic, so a word is either
// empty or complete: the reader polls the data itself, no flag and no fence, and puts MAILBOX_EMPTY back when it has read it.
// The all-ones pattern is a NaN no arithmetic produces (results that are NaN travel as the canonical quiet NaN).
constexpr uint32_t MAILBOX_EMPTY = 0xFFFFFFFFu;
__device__ __forceinline__ uint32_t mailbox_bits(float v) { const uint32_t b = __float_as_uint(v); return b == MAILBOX_EMPTY ? 0x7FC00000u : b; }
__device__ __forceinline__ void mailbox_store(uint32_t* p, uint32_t bits) { asm volatile("st.relaxed.sys.global.u32 [%0], %1;" ::"l"(p), "r"(bits) : "memory"); }
__device__ __forceinline__ uint32_t mailbox_load(const uint32_t* p) {
  uint32_t v;
  asm volatile("ld.relaxed.sys.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}

// One thread of a converged warp.  A producer or MMA thread is elected, not taken as `lane == 0`: under elect.sync the compiler may use
// uniform registers, which the tcgen05, bulk-copy and barrier instructions take their operands from.  As plain `lane == 0` code an MMA thread
// needed 80 cycles to issue an instruction and over 300 for a barrier that was ready (many-row GEMM, 8B gate/up, 8 rows: 127 -> 90 us).
__device__ __forceinline__ bool elect_one() {
  uint32_t e;
  asm volatile("{\n.reg .pred p;\nelect.sync _|p, 0xffffffff;\nselp.u32 %0, 1, 0, p;\n}" : "=r"(e));
  return e != 0;
}

// Ask for a line that will be read behind pdl_wait (weights, tables): in a model whose weights exceed L2 it is a DRAM miss by then.
__device__ __forceinline__ void prefetch_l2(const void* p) { asm volatile("prefetch.global.L2 [%0];" ::"l"(p)); }

// ---- thread-block clusters ----
__device__ __forceinline__ float ld_cluster(uint32_t local, uint32_t rank) {      // the same shared-memory word of another CTA of the cluster
  uint32_t a;
  float v;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"(local), "r"(rank));
  asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v) : "r"(a) : "memory");
  return v;
}
__device__ __forceinline__ void cluster_arrive() { asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory"); }
__device__ __forceinline__ void cluster_wait() { asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory"); }
__device__ __forceinline__ void cluster_sync() { cluster_arrive(); cluster_wait(); }

// The power of two that puts a largest magnitude into [2^13, 2^14), where fp16 holds a value and the remainder's rounding to 2^-22 of it and to 2^-38 of
// the largest, and its inverse; zeros get the inverse 0, infinities (and NaN) are left as they are.
__device__ __forceinline__ void pow2_scale(float amax, float& up, float& down) {
  const int e = max((int)(__float_as_uint(amax) >> 23) - 127, -100);
  const bool live = amax > 0.f && amax < INFINITY;
  up = live ? __uint_as_float((uint32_t)(13 - e + 127) << 23) : 1.f;
  down = live ? __uint_as_float((uint32_t)(e - 13 + 127) << 23) : amax > 0.f ? 1.f : 0.f;
}

__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}
__device__ __forceinline__ float warp_max(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
  return v;
}

__device__ __forceinline__ uint4 ldg_stream(const uint4* p) {   // weights are read once: do not keep them in L1
  uint4 v;
  asm volatile("ld.global.nc.L1::no_allocate.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p));
  return v;
}
__device__ __forceinline__ uint2 ldg_stream(const uint2* p) {
  uint2 v;
  asm volatile("ld.global.nc.L1::no_allocate.v2.u32 {%0,%1}, [%2];" : "=r"(v.x), "=r"(v.y) : "l"(p));
  return v;
}
