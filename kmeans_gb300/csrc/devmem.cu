// Device memory: two stream-ordered memory pools per device, owned by the library.
//
// Handles. A handle's fixed buffers are one arena (engine.cu). With cudaMalloc/cudaFree a one-shot call
// on the 4M x 128, K=1024 workload spent ~1 ms allocating and ~3.3 ms freeing its ~7 GB (the
// free synchronizes the device and unmaps). Here the arena comes from a pool whose release
// threshold is unbounded: cudaFreeAsync hands the memory back to the pool, and the next handle
// of the same or a smaller size takes it again without mapping anything. The pool keeps what it
// holds until kmgb_release_cached_memory() (or a failed allocation, which trims both pools and retries
// once); KMGB_POOL=0 trims after every free, which gives back cudaMalloc/cudaFree behaviour.
//
// Calls (computeKmeansD, batched problems, kmgb_kmeanspp_*, ClosestCenters). Their workspaces come from
// a pool of their own that keeps at most kCallPoolKeep between them: what it holds beyond goes back to
// the device with the next synchronization after the call (KMGB_POOL=0: all of it). So a call neither
// leaves a large workspace behind nor unmaps what handles have cached.
#include <cuda_runtime.h>

#include <atomic>
#include <cstdint>
#include <cstdlib>
#include <cstring>
#include <mutex>

#include "../../include/kmeans_gb300.h"
#include "kernels.h"

namespace kmgb {
namespace {

constexpr int kMaxDevices = 64;
std::mutex g_mu;
constexpr int kHandles = 0, kCalls = 1;
constexpr uint64_t kCallPoolKeep = 8ull << 30;
cudaMemPool_t g_pools[2][kMaxDevices] = {};

bool keep_freed_memory() {
  static const bool keep = [] {
    const char* v = std::getenv("KMGB_POOL");
    return !(v && std::strcmp(v, "0") == 0);
  }();
  return keep;
}

cudaError_t pool_of_current_device(int kind, cudaMemPool_t* out) {
  int dev = 0;
  cudaError_t r = cudaGetDevice(&dev);
  if (r != cudaSuccess) return r;
  if (dev < 0 || dev >= kMaxDevices) return cudaErrorInvalidDevice;
  std::lock_guard<std::mutex> g(g_mu);
  if (!g_pools[kind][dev]) {
    cudaMemPoolProps props;
    std::memset(&props, 0, sizeof(props));
    props.allocType = cudaMemAllocationTypePinned;
    props.handleTypes = cudaMemHandleTypeNone;
    props.location.type = cudaMemLocationTypeDevice;
    props.location.id = dev;
    cudaMemPool_t p = nullptr;
    r = cudaMemPoolCreate(&p, &props);
    if (r != cudaSuccess) return r;
    uint64_t threshold = kind == kHandles ? UINT64_MAX : keep_freed_memory() ? kCallPoolKeep : 0;
    r = cudaMemPoolSetAttribute(p, cudaMemPoolAttrReleaseThreshold, &threshold);
    if (r != cudaSuccess) {
      cudaMemPoolDestroy(p);
      return r;
    }
    g_pools[kind][dev] = p;
  }
  *out = g_pools[kind][dev];
  return cudaSuccess;
}

}  // namespace

// Test hooks: a countdown per event kind; the event that brings it to zero fails once.
std::atomic<long long> g_fail_countdown[4];
std::atomic<long long> g_test_withhold{0};
std::atomic<unsigned long long> g_test_wait{0};

bool inject_fault(int kind) {
  if (kind < 1 || kind > 3) return false;
  long long v = g_fail_countdown[kind].load(std::memory_order_relaxed);
  while (v > 0) {
    if (g_fail_countdown[kind].compare_exchange_weak(v, v - 1, std::memory_order_relaxed))
      return v == 1;
  }
  return false;
}

void test_wait_hook(long long* withhold, unsigned long long* wait_cycles) {
  *withhold = g_test_withhold.load(std::memory_order_relaxed);
  *wait_cycles = g_test_wait.load(std::memory_order_relaxed);
}

int num_sms() {
  static std::atomic<int> cached[kMaxDevices];
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kMaxDevices) return 148;
  int v = cached[dev].load(std::memory_order_relaxed);
  if (v <= 0) {
    if (cudaDeviceGetAttribute(&v, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || v <= 0)
      v = 148;  // any positive count only sizes grids; every kernel strides over its work
    cached[dev].store(v, std::memory_order_relaxed);
  }
  return v;
}

static cudaError_t alloc_from(int kind, void** p, size_t bytes, cudaStream_t s) {
  *p = nullptr;
  if (inject_fault(kFaultAlloc)) return cudaErrorMemoryAllocation;
  if (bytes == 0) bytes = 1;
  cudaMemPool_t pool[2] = {nullptr, nullptr};
  for (int i = 0; i < 2; ++i) {
    const cudaError_t r = pool_of_current_device(i, &pool[i]);
    if (r != cudaSuccess) return r;
  }
  cudaError_t r = cudaMallocFromPoolAsync(p, bytes, pool[kind], s);
  if (r == cudaErrorMemoryAllocation) {
    // memory the pools hold but nobody uses goes back to the device, then one more try
    cudaGetLastError();
    cudaDeviceSynchronize();
    for (cudaMemPool_t q : pool) cudaMemPoolTrimTo(q, 0);
    r = cudaMallocFromPoolAsync(p, bytes, pool[kind], s);
  }
  if (r != cudaSuccess) *p = nullptr;
  return r;
}

cudaError_t dev_alloc(void** p, size_t bytes, cudaStream_t s) {
  const cudaError_t r = alloc_from(kHandles, p, bytes, s);
  if (r != cudaSuccess) return r;
  // usable from every stream (copies on the legacy stream, a handle's copy stream) at once
  return cudaStreamSynchronize(s);
}

void dev_free(void* p, cudaStream_t s) {
  if (!p) return;
  cudaFreeAsync(p, s);
  if (!keep_freed_memory()) {
    cudaStreamSynchronize(s);
    cudaMemPool_t pool = nullptr;
    if (pool_of_current_device(kHandles, &pool) == cudaSuccess) cudaMemPoolTrimTo(pool, 0);
  }
}

cudaError_t call_alloc(void** p, size_t bytes, cudaStream_t s) { return alloc_from(kCalls, p, bytes, s); }

void call_free(void* p, cudaStream_t s) {
  if (p) cudaFreeAsync(p, s);
}

size_t dev_available() {
  size_t mem_free = 0, mem_total = 0;
  if (cudaMemGetInfo(&mem_free, &mem_total) != cudaSuccess) {
    cudaGetLastError();
    return 0;
  }
  for (int kind = 0; kind < 2; ++kind) {
    cudaMemPool_t pool = nullptr;
    uint64_t held = 0, used = 0;
    if (pool_of_current_device(kind, &pool) == cudaSuccess &&
        cudaMemPoolGetAttribute(pool, cudaMemPoolAttrReservedMemCurrent, &held) == cudaSuccess &&
        cudaMemPoolGetAttribute(pool, cudaMemPoolAttrUsedMemCurrent, &used) == cudaSuccess && held > used)
      mem_free += held - used;
  }
  return mem_free;
}

cudaError_t dev_release_cached() {
  cudaError_t r = cudaDeviceSynchronize();
  std::lock_guard<std::mutex> g(g_mu);
  for (auto& pools : g_pools)
    for (cudaMemPool_t p : pools)
      if (p) {
        const cudaError_t t = cudaMemPoolTrimTo(p, 0);
        if (r == cudaSuccess) r = t;
      }
  return r;
}

}  // namespace kmgb

extern "C" {

void kmgb_debug_fail_nth(int kind, long long nth) {
  if (kind < 1 || kind > 3) return;
  kmgb::g_fail_countdown[kind].store(nth > 0 ? nth : 0, std::memory_order_relaxed);
}

void kmgb_debug_withhold_stage(long long stage, unsigned long long wait_cycles) {
  kmgb::g_test_withhold.store(stage > 0 ? stage : 0, std::memory_order_relaxed);
  kmgb::g_test_wait.store(stage > 0 ? wait_cycles : 0, std::memory_order_relaxed);
}

long long kmgb_debug_pool_used_bytes(void) {
  long long sum = 0;
  for (int kind = 0; kind < 2; ++kind) {
    cudaMemPool_t pool = nullptr;
    uint64_t used = 0;
    if (kmgb::pool_of_current_device(kind, &pool) != cudaSuccess ||
        cudaMemPoolGetAttribute(pool, cudaMemPoolAttrUsedMemCurrent, &used) != cudaSuccess)
      return -1;
    sum += (long long)used;
  }
  return sum;
}

int kmgb_release_cached_memory(void) {
  const cudaError_t r = kmgb::dev_release_cached();
  if (r != cudaSuccess) {
    kmgb::set_last_error(cudaGetErrorString(r));
    return 1;
  }
  return 0;
}

}  // extern "C"
