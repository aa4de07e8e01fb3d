// Results that are allocated on every call (QuantLinear, FP8Linear, dequantize): a pool of device blocks and the one-call Linear on top of it.
//
// What it replaces: cudaMalloc / cudaFree per result.  cudaFree waits for the whole device and both change the address space: 0.1 to 2 ms
// per call with megabyte results, against kernels of 10 to 60 us.
//
// A freed block may still be read by work that was queued before, on any stream, ours or a caller's, and the library cannot know which.
// cudaFree's own guarantee is kept: a block is handed out again only after the device has been seen idle (one cudaDeviceSynchronize) at some
// time after it was freed.  Freed blocks wait in a list; when the list holds PENDING_BLOCKS blocks or PENDING_BYTES, the next allocation
// waits for the device once and turns the whole list into free blocks.  So a loop of calls waits once per 64 results (or 64 MiB) instead of
// once per result.  Bounded: at most POOL_BYTES are kept per device (past that everything unused goes back with cudaFree), larger blocks than
// BLOCK_MAX never enter, and everything goes back when an allocation fails or b200q_pool_trim is called.  Any thread may call.  A device's lists have a lock
// of their own, held during its wait: work on one device may depend on a thread that is allocating on another.
#include "common.cuh"
#include <mutex>
#include <new>
#include <unordered_map>
#include <vector>

namespace {

constexpr size_t BLOCK_MAX = (size_t)32 << 20, POOL_BYTES = (size_t)256 << 20, PENDING_BYTES = (size_t)64 << 20;
constexpr size_t PENDING_BLOCKS = 64;

struct Block { void* p; size_t size; };
struct DevicePool {
  std::unordered_map<size_t, std::vector<void*>> free_;       // by size
  std::vector<Block> pending;
  size_t pending_bytes = 0, kept = 0;                          // kept: free and pending bytes
  std::mutex lock;
};
DevicePool g_pool[B200Q_MAX_DEVICES];
std::mutex g_out_lock;                                         // never held together with a device's
std::unordered_map<void*, std::pair<int, size_t>> g_out;      // blocks in use: device, size (0: not a pool size)

// sizes in steps of an eighth of a power of two: at most an eighth is lost, and few sizes occur
size_t round_size(size_t n) {
  if (n < 512) return 512;
  size_t step = 64;
  while (step * 16 < n) step *= 2;
  return (n + step - 1) / step * step;
}

cudaError_t recycle(DevicePool& d) {                           // after this every pending block is free
  const cudaError_t e = cudaDeviceSynchronize();
  if (e != cudaSuccess) return e;
  while (!d.pending.empty()) {                                 // one by one: a block is in one list at any time, whatever is thrown
    const Block b = d.pending.back();
    d.free_[b.size].push_back(b.p);
    d.pending.pop_back();
    d.pending_bytes -= b.size;
  }
  return cudaSuccess;
}

void give_back(DevicePool& d) {                                // cudaFree waits for the device itself
  for (const Block& b : d.pending) cudaFree(b.p);
  d.pending.clear();
  for (auto& f : d.free_)
    for (void* p : f.second) cudaFree(p);
  d.free_.clear();
  d.pending_bytes = d.kept = 0;
}

int take_block(DevicePool& d, void** out, size_t size) {
  std::lock_guard<std::mutex> g(d.lock);
  if (d.pending.size() >= PENDING_BLOCKS || d.pending_bytes >= PENDING_BYTES) B200Q_CHECK_CUDA(recycle(d));
  auto it = d.free_.find(size);
  if (it != d.free_.end() && !it->second.empty()) {
    *out = it->second.back();
    it->second.pop_back();
    d.kept -= size;
    return B200Q_OK;
  }
  cudaError_t e = cudaMalloc(out, size);
  if (e == cudaErrorMemoryAllocation) {
    cudaGetLastError();
    give_back(d);
    e = cudaMalloc(out, size);
  }
  B200Q_CHECK_CUDA(e);
  return B200Q_OK;
}

// A result of work that is being captured belongs to the graph, which may write it long after it was freed here: it is no block of the pool but an allocation
// of its own, which most capture modes refuse, as they do for any caller.
int pool_alloc(void** out, size_t bytes, cudaStream_t st) {
  const int dev = b200q_current_device();
  if (dev < 0) return B200Q_ERR_CUDA;
  cudaStreamCaptureStatus capture = cudaStreamCaptureStatusNone;
  if (cudaStreamIsCapturing(st, &capture) != cudaSuccess) cudaGetLastError();      // the legacy stream beside a capture: not captured itself
  const bool pooled = bytes <= BLOCK_MAX && capture == cudaStreamCaptureStatusNone;
  const size_t size = pooled ? round_size(bytes) : bytes ? bytes : 1;
  if (pooled) {
    const int rc = take_block(g_pool[dev], out, size);
    if (rc != B200Q_OK) return rc;
  } else {
    const int rc = b200q_malloc(out, size);
    if (rc != B200Q_OK) return rc;
  }
  try {
    std::lock_guard<std::mutex> g(g_out_lock);
    g_out[*out] = {dev, pooled ? size : 0};
  } catch (...) {
    cudaFree(*out);
    *out = nullptr;
    throw;
  }
  return B200Q_OK;
}
// Nothing is thrown across the C interface: the lists need host memory, and there may be none.
template <typename F> int guarded(const F& f) {
  try { return f(); } catch (const std::bad_alloc&) {
    b200q_set_cuda_error(cudaErrorMemoryAllocation);
    return B200Q_ERR_CUDA;
  }
}

}  // namespace

// called when an ordinary allocation fails: true if there was something to give back
bool b200q_pool_release(int dev) {
  std::lock_guard<std::mutex> g(g_pool[dev].lock);
  const bool any = g_pool[dev].kept > 0;
  give_back(g_pool[dev]);
  return any;
}

extern "C" int b200q_pool_alloc(void** device_ptr, size_t bytes, void* stream) {
  return device_ptr ? guarded([&] { return pool_alloc(device_ptr, bytes, (cudaStream_t)stream); }) : B200Q_ERR_BAD_ARG;
}

extern "C" int b200q_pool_free(void* device_ptr) {
  if (!device_ptr) return B200Q_OK;
  int dev;
  size_t size;
  {
    std::lock_guard<std::mutex> g(g_out_lock);
    auto it = g_out.find(device_ptr);
    if (it == g_out.end()) return B200Q_ERR_BAD_ARG;
    dev = it->second.first; size = it->second.second;
    g_out.erase(it);
  }
  if (size) {
    DevicePool& d = g_pool[dev];
    std::lock_guard<std::mutex> g(d.lock);
    if (d.kept + size > POOL_BYTES) give_back(d);              // full of blocks that nobody has asked for lately
    const bool kept = guarded([&] { d.pending.push_back({device_ptr, size}); return B200Q_OK; }) == B200Q_OK;
    if (kept) {
      d.pending_bytes += size;
      d.kept += size;
      return B200Q_OK;
    }
  }
  B200Q_CHECK_CUDA(cudaFree(device_ptr));
  return B200Q_OK;
}

extern "C" int b200q_pool_trim(void) {
  const int dev = b200q_current_device();
  if (dev < 0) return B200Q_ERR_CUDA;
  b200q_pool_release(dev);
  return B200Q_OK;
}

// y = Linear(x) with the result in a new pool block: QuantLinear.__call__ in one call across the language border.
extern "C" int b200q_linear(const b200q_linear_desc* l, const void* x, int dtype, int m, void** y, void* stream) {
  if (!l || !y || m < 0 || (dtype != B200Q_F32 && dtype != B200Q_F16) || (m && !x)) return B200Q_ERR_BAD_ARG;
  const size_t row = (size_t)l->n_out * (dtype == B200Q_F32 ? 4 : 2);
  int rc = b200q_pool_alloc(y, (size_t)m * row, stream);
  if (rc != B200Q_OK || m == 0) return rc;
  if (l->dense) rc = b200q_gemv_dense(l->w, l->w_type, l->n_out, l->n_in, m, x, dtype, nullptr, 0.f, l->bias, nullptr, *y, dtype, 0, stream);
  else if (m >= l->gemm_min_rows && l->w_type != B200Q_Q6_K)
    rc = b200q_qgemm_ws(l->w_type, l->w, x, dtype, l->bias, nullptr, B200Q_EPI_LINEAR, *y, dtype, m, l->n_out, l->n_in, l->workspace, l->workspace_bytes, stream);
  else {
    b200q_gemv_args a = {};
    a.qtype = l->w_type; a.n_out = l->n_out; a.n_in = l->n_in; a.m = m; a.w_packed = l->w; a.x = x; a.x_dtype = dtype; a.y_dtype = dtype;
    a.epilogue = B200Q_EPI_LINEAR; a.bias = l->bias; a.y = *y; a.residual_scale = 1.f;
    rc = b200q_gemv(&a, stream);
  }
  if (rc != B200Q_OK) { b200q_pool_free(*y); *y = nullptr; }
  return rc;
}
