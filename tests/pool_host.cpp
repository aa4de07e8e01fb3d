// The result pool (csrc/pool.cu) on a made-up device: the CUDA calls it makes are answered here, so its rules can be checked without a GPU.
#include <cuda_runtime.h>
#include <atomic>
#include <chrono>
#include <cstdio>
#include <cstdlib>
#include <new>
#include <set>
#include <thread>
#include "../include/b200q.h"

static thread_local int g_device = 0;
static std::atomic<int> g_syncs[2], g_mallocs, g_frees;
static cudaStreamCaptureStatus g_capture = cudaStreamCaptureStatusNone;
static std::atomic<bool> g_hold{false}, g_held{false};       // device 0's synchronisation waits while g_hold is set
static char g_bytes[1 << 16];
static bool g_full = false;                                  // host memory has run out

void* operator new(size_t n) {
  if (g_full) throw std::bad_alloc();
  return malloc(n);
}
void operator delete(void* p) noexcept { free(p); }
void operator delete(void* p, size_t) noexcept { free(p); }

extern "C" {
cudaError_t cudaStreamIsCapturing(cudaStream_t st, cudaStreamCaptureStatus* s) { *s = st ? g_capture : cudaStreamCaptureStatusNone; return cudaSuccess; }
cudaError_t cudaMalloc(void** p, size_t) {
  static std::atomic<int> n{0};
  *p = g_bytes + 16 * n++;
  g_mallocs++;
  return cudaSuccess;
}
cudaError_t cudaFree(void*) { g_frees++; return cudaSuccess; }
cudaError_t cudaDeviceSynchronize() {
  g_syncs[g_device]++;
  if (g_device == 0) while (g_hold) { g_held = true; std::this_thread::yield(); }
  return cudaSuccess;
}
cudaError_t cudaGetLastError() { return cudaSuccess; }
int b200q_gemv(const b200q_gemv_args*, void*) { return 0; }
int b200q_gemv_dense(const void*, int, int, int, int, const void*, int, const void*, float, const void*, const void*, void*, int, int, void*) { return 0; }
int b200q_qgemm_ws(int, const void*, const void*, int, const void*, const void*, int, void*, int, int, int, int, void*, size_t, void*) { return 0; }
}
void b200q_set_cuda_error(cudaError_t) {}
int b200q_current_device() { return g_device; }
extern "C" int b200q_malloc(void** p, size_t n) { return cudaMalloc(p, n) == cudaSuccess ? 0 : B200Q_ERR_CUDA; }

#define CHECK(c) do { if (!(c)) { printf("line %d: %s\n", __LINE__, #c); exit(1); } } while (0)
static void* get(size_t n, void* st = nullptr) { void* p = nullptr; CHECK(b200q_pool_alloc(&p, n, st) == 0); return p; }

int main() {
  // a freed block comes back only after the device has been waited for since
  void* a = get(4096);
  CHECK(b200q_pool_free(a) == 0);
  std::set<void*> seen;
  for (int i = 0; i < 70; i++) {
    const int syncs = g_syncs[0];
    void* p = get(4096);
    CHECK((p != a && !seen.count(p)) || g_syncs[0] > 0);
    if (g_syncs[0] != syncs) seen.clear();               // everything freed before that wait may be handed out again
    CHECK(b200q_pool_free(p) == 0);
    seen.insert(p);
  }
  CHECK(g_syncs[0] == 1 && g_mallocs < 70);              // one wait for 64 blocks
  // sizes are rounded up by an eighth at most, large blocks and trimmed ones go back to the device
  const int frees = g_frees;
  void* big = get((size_t)33 << 20);
  CHECK(b200q_pool_free(big) == 0 && g_frees == frees + 1);
  CHECK(b200q_pool_trim() == 0 && g_frees > frees + 1);
  CHECK(b200q_pool_free((char*)a + 8) == B200Q_ERR_BAD_ARG);
  // what a captured stream is to write comes from no pool and goes back to none
  CHECK(b200q_pool_free(get(4096)) == 0);
  for (int i = 0; i < 64; i++) CHECK(b200q_pool_free(get(8192)) == 0);      // the next block of the pool is one that was in use
  g_capture = cudaStreamCaptureStatusActive;
  const int syncs = g_syncs[0], mallocs = g_mallocs, freed = g_frees;
  void* c = get(4096, (void*)1);
  CHECK(g_syncs[0] == syncs && g_mallocs == mallocs + 1);
  CHECK(b200q_pool_free(c) == 0 && g_frees == freed + 1);
  g_capture = cudaStreamCaptureStatusNone;
  CHECK(b200q_pool_trim() == 0);
  // no host memory: an error, no exception, and no block lost or handed out twice
  std::set<void*> out, blocks;
  for (int i = 0; i < 40; i++) blocks.insert(get(1024));
  for (void* p : blocks) CHECK(b200q_pool_free(p) == 0);
  const int given = g_mallocs, returned = g_frees;
  void* none = nullptr;
  g_full = true;
  CHECK(b200q_pool_alloc(&none, 2048, nullptr) == B200Q_ERR_CUDA);
  g_full = false;
  CHECK(g_mallocs - given == g_frees - returned);
  for (int i = 0; i < 60; i++) CHECK(b200q_pool_free(get(512 + 512 * (i & 7))) == 0);
  for (int i = 0; i < 200; i++) { void* p = get(1024); CHECK(out.insert(p).second); }
  for (void* p : out) CHECK(b200q_pool_free(p) == 0);
  CHECK(b200q_pool_trim() == 0);
  // one device's wait stops nobody on another
  for (int i = 0; i < 64; i++) CHECK(b200q_pool_free(get(512)) == 0);      // no free block, 64 that wait
  g_hold = true;
  std::thread t([] { void* p = nullptr; b200q_pool_alloc(&p, 512, nullptr); });
  for (int i = 0; !g_held && i < 10000; i++) std::this_thread::sleep_for(std::chrono::milliseconds(1));
  CHECK(g_held);
  std::atomic<bool> done{false};
  std::thread u([&] { g_device = 1; void* p = nullptr; done = b200q_pool_alloc(&p, 512, nullptr) == 0 && b200q_pool_free(p) == 0; });
  for (int i = 0; !done && i < 2000; i++) std::this_thread::sleep_for(std::chrono::milliseconds(1));
  const bool other = done;
  g_hold = false;
  t.join(); u.join();
  CHECK(other);
  printf("ok\n");
  return 0;
}
