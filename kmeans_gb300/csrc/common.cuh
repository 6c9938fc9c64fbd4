// Shared device/host helpers for the GB300 (sm_103a) Lloyd kernels.
//
// Every wait on an mbarrier is bounded: a wait gives up after KMGB_WAIT_CYCLES SM clock cycles
// (about 2 s at 2 GHz), records an error code in the launch's error word and returns false; an
// abort flag in shared memory then makes every later wait of the CTA return at once so the CTA
// drains and exits (no unbounded spin, no __trap). The limit is counted with clock64, a cheap
// register read: a %globaltimer read takes hundreds of cycles on GB300 and, inside the wait
// loop, delayed every wake-up of the pipelines by about that much.
#pragma once

#include <cuda.h>
#include <cuda_runtime.h>
#include <cuda_bf16.h>
#include <stdint.h>

#include <utility>

#ifndef KMGB_WAIT_CYCLES
#define KMGB_WAIT_CYCLES 4000000000ull  // about 2 s per wait at a 2 GHz SM clock
#endif

// Error codes written to the device error word (first writer wins).
enum kmgb_dev_error {
  KMGB_DEV_OK = 0,
  KMGB_DEV_TIMEOUT_FULL = 1,     // consumer waited too long for a TMA stage
  KMGB_DEV_TIMEOUT_EMPTY = 2,    // producer waited too long for a free stage
  KMGB_DEV_TIMEOUT_ACC = 3,      // MMA / epilogue accumulator hand-off timed out
  KMGB_DEV_BAD_LABEL = 4,        // a label outside [0, K) reached the update
  KMGB_DEV_BAD_SHAPE = 5,
};

namespace kmgb {

__device__ __forceinline__ uint32_t smem_u32(const void* p) {
  return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}

__device__ __forceinline__ void set_error(int* err, int code) {
  if (err) atomicCAS(err, 0, code);
}

__device__ __forceinline__ void mbar_init(uint32_t bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count) : "memory");
}

__device__ __forceinline__ void fence_mbar_init() {
  asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}

__device__ __forceinline__ void fence_proxy_async() {
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
}

__device__ __forceinline__ void mbar_arrive(uint32_t bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}

__device__ __forceinline__ void mbar_arrive_expect_tx(uint32_t bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes)
               : "memory");
}

__device__ __forceinline__ bool mbar_try_wait(uint32_t bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(ok)
      : "r"(bar), "r"(parity)
      : "memory");
  return ok != 0;
}

// Bounded wait. `abort_flag` is a CTA-shared word: once set, waits return false at once.
// `limit`: SM cycles before giving up (KMGB_WAIT_CYCLES unless a test shortens it).
__device__ __forceinline__ bool mbar_wait(uint32_t bar, uint32_t parity, volatile int* abort_flag,
                                          int* err, int code,
                                          unsigned long long limit = KMGB_WAIT_CYCLES) {
  if (mbar_try_wait(bar, parity)) return true;
  const long long t0 = clock64();
  while (true) {
    if (mbar_try_wait(bar, parity)) return true;
    if (*abort_flag) return false;
    if ((unsigned long long)(clock64() - t0) > limit) {
      *abort_flag = 1;
      set_error(err, code);
      return false;
    }
  }
}

// 2-D TMA tile load into shared memory, completion signalled on `bar` (complete_tx bytes).
__device__ __forceinline__ void tma_load_2d(uint32_t dst, const CUtensorMap* map, uint32_t bar,
                                            int c0, int c1) {
  asm volatile(
      "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes"
      " [%0], [%1, {%3, %4}], [%2];" ::"r"(dst),
      "l"(reinterpret_cast<uint64_t>(map)), "r"(bar), "r"(c0), "r"(c1)
      : "memory");
}

__device__ __forceinline__ void prefetch_tmap(const CUtensorMap* map) {
  asm volatile("prefetch.tensormap [%0];" ::"l"(reinterpret_cast<uint64_t>(map)) : "memory");
}

// Byte offset of the 16-byte chunk `chunk` of row `row` inside a tile written by TMA with
// CU_TENSOR_MAP_SWIZZLE_128B (rows of 128 bytes, tile base 1024-byte aligned): the chunk index
// is XOR-ed with the row index modulo 8.
__device__ __forceinline__ uint32_t swz128(uint32_t row, uint32_t chunk) {
  return row * 128u + ((chunk ^ (row & 7u)) << 4);
}

// First statement of every kernel that launch() starts: waits until the grids before it in its stream
// are complete and their writes visible, then lets the next grid's blocks take their places. Returns
// false; the compiler cannot know it, so that no load moves above the wait.
__device__ __forceinline__ bool grid_enter() {
  unsigned z;
  asm volatile("griddepcontrol.wait;\n\tmov.u32 %0, 0;" : "=r"(z) : : "memory");
  asm volatile("griddepcontrol.launch_dependents;" : : : "memory");
  return z != 0;
}

// Kernels load global memory through coherent loads: one that launch() starts may begin while the grid
// before it still writes, so what that grid writes is not read-only for the kernel's lifetime, as __ldg and
// const __restrict__ kernel parameters (which the compiler turns into the same instruction) require.
// grid_enter() orders the loads after the grid's end and, for coherent loads, makes its writes visible.
// ld: one that stays in its place among the others, ahead of what is written after it (free to move, loads
// for the next step of a loop ended up behind the work they were to overlap).
__device__ __forceinline__ void ld_to(const int* p, int& v) {
  asm volatile("ld.global.b32 %0, [%1];" : "=r"(v) : "l"(p));
}
__device__ __forceinline__ void ld_to(const float* p, float& v) {
  asm volatile("ld.global.f32 %0, [%1];" : "=f"(v) : "l"(p));
}
__device__ __forceinline__ void ld_to(const double* p, double& v) {
  asm volatile("ld.global.f64 %0, [%1];" : "=d"(v) : "l"(p));
}
__device__ __forceinline__ void ld_to(const float4* p, float4& v) {
  asm volatile("ld.global.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "l"(p));
}
__device__ __forceinline__ void ld_to(const uint4* p, uint4& v) {
  asm volatile("ld.global.v4.b32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p));
}
__device__ __forceinline__ void ld_to(const double2* p, double2& v) {
  asm volatile("ld.global.v2.f64 {%0, %1}, [%2];" : "=d"(v.x), "=d"(v.y) : "l"(p));
}
template <typename T>
__device__ __forceinline__ T ld(const T* p) {
  T v;
  ld_to(p, v);
  return v;
}

// Rows list[slot], slot < cnt, of one or two planes of row_vec 16-byte vectors a row, into rows `slot` of
// their compact copies, by the warps w0, w0 + nw, ... (16 bytes a lane). Four loads a lane stand ahead of
// their stores, which a coherent load does not pass: 86 us an iteration (mean of the first four) of
// 4M x 128, K=1024; 151 with a load and a store at a time, 123 with the non-coherent loads that the
// compiler moved ahead itself.
__device__ __forceinline__ void copy_listed_rows(const int* list, long long cnt, const uint4* Xb,
                                                 const uint4* Xl, int row_vec, uint4* XbC, uint4* XlC,
                                                 long long w0, long long nw, int lane) {
  const int per = Xl ? 2 * row_vec : row_vec;
  if (per <= 32) {  // 32 / per rows a step, four steps together
    constexpr int U = 4;
    const int rows = 32 / per, rr = lane / per, v = lane - rr * per;
    const uint4* src = v < row_vec ? Xb + v : Xl + (v - row_vec);
    uint4* dst = v < row_vec ? XbC + v : XlC + (v - row_vec);
    for (long long s0 = w0 * rows * U; s0 < cnt; s0 += nw * rows * U) {
      int pt[U];
      uint4 x[U];
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const long long slot = s0 + u * rows + rr;
        pt[u] = ld(list + (slot < cnt ? slot : cnt - 1));
      }
#pragma unroll
      for (int u = 0; u < U; ++u) x[u] = ld(src + (size_t)pt[u] * row_vec);
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const long long slot = s0 + u * rows + rr;
        if (rr < rows && slot < cnt) dst[(size_t)slot * row_vec] = x[u];
      }
    }
    return;
  }
  for (long long s0 = 2 * w0; s0 < cnt; s0 += 2 * nw) {  // two rows, two vectors of each
    const bool two = s0 + 1 < cnt;
    const size_t p0 = (size_t)ld(list + s0) * row_vec, p1 = (size_t)ld(list + s0 + two) * row_vec;
    const size_t d0 = (size_t)s0 * row_vec, d1 = d0 + row_vec;
    for (int v0 = lane; v0 < per; v0 += 64) {
      const bool more = v0 + 32 < per;
      const int v1 = more ? v0 + 32 : v0;
      const uint4* a = v0 < row_vec ? Xb + v0 : Xl + (v0 - row_vec);
      const uint4* b = v1 < row_vec ? Xb + v1 : Xl + (v1 - row_vec);
      uint4* ao = v0 < row_vec ? XbC + v0 : XlC + (v0 - row_vec);
      uint4* bo = v1 < row_vec ? XbC + v1 : XlC + (v1 - row_vec);
      const uint4 x0 = ld(a + p0), x1 = ld(a + p1), y0 = ld(b + p0), y1 = ld(b + p1);
      ao[d0] = x0;
      if (two) ao[d1] = x1;
      if (more) bo[d0] = y0;
      if (more && two) bo[d1] = y1;
    }
  }
}

// A load that stays where it is written, ahead of the test of a flag loaded with it: one after the
// other, the flags and counts at a kernel's start cost a round trip to L2 (900 cycles) each. It goes
// through L1 (a volatile load of one word by every warp of a large grid does not: 6.8 -> 13.3 us for two
// words and 10,000 warps); the words are written by earlier grids only.
__device__ __forceinline__ int pinned(const int* p) {
  int v;
  asm volatile("ld.global.b32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}

// Device-side stop rule of the Lloyd loop: once the flag is set every later kernel of the run
// returns at once, so the host never has to synchronise to evaluate the criterion.
__device__ __forceinline__ bool stopped(const int* stop) { return stop != nullptr && pinned(stop) != 0; }

__device__ __forceinline__ unsigned lanemask_lt() {
  unsigned m;
  asm("mov.u32 %0, %%lanemask_lt;" : "=r"(m));
  return m;
}

// Bits of a label below k (0 for k <= 1).
__device__ __forceinline__ int label_bits(int k) { return k <= 1 ? 0 : 32 - __clz(k - 1); }

// The lanes of the warp holding the same label as this lane (labels in [0, 2^nbits), or -1 for
// "none": the -1 lanes form one group of their own). One ballot per label bit: with mostly
// distinct labels in a warp (K ~ 1000 centers) this is much cheaper than __match_any_sync.
// Every lane of the warp calls it with the same nbits.
__device__ __forceinline__ unsigned warp_peers(int l, int nbits) {
  const unsigned valid = __ballot_sync(0xffffffffu, l >= 0);
  unsigned m = l >= 0 ? valid : ~valid;
  for (int b = 0; b < nbits; ++b) {
    const bool bit = (l >> b) & 1;
    const unsigned set = __ballot_sync(0xffffffffu, bit);
    m &= bit ? set : ~set;
  }
  return m;
}

}  // namespace kmgb

// Host-side: 2-D row-major tensor map (inner dim = columns) with 128-byte swizzle.
// dtype: CU_TENSOR_MAP_DATA_TYPE_FLOAT32 or _BFLOAT16. Returns cudaSuccess or an error.
cudaError_t kmgb_make_tmap_2d(CUtensorMap* map, const void* base, CUtensorMapDataType dtype,
                              int elem_bytes, uint64_t cols, uint64_t rows, uint64_t row_stride_bytes,
                              uint32_t box_cols, uint32_t box_rows);
// The same with a given swizzle (the box's inner extent at most the swizzle width; without one, 256
// elements).
cudaError_t kmgb_make_tmap_2d_swz(CUtensorMap* map, const void* base, CUtensorMapDataType dtype,
                                  int elem_bytes, uint64_t cols, uint64_t rows,
                                  uint64_t row_stride_bytes, uint32_t box_cols, uint32_t box_rows,
                                  CUtensorMapSwizzle swizzle);

// Number of kernels this library has launched (process-wide), for launch accounting.
namespace kmgb {
void count_launches(long long n);
long long launch_count();
long long thread_launch_count();  // of the calling thread: what its captured graph holds
// Whether a launch may overlap the grid before it in its stream (programmatic dependent launch): its
// blocks take their places while that grid still runs and wait in grid_enter() for its end. Launches
// one by one gain by it -- five short kernels an entry of the per-kernel interface on 100,000 x 64,
// K=256 (FP64): 0.78 -> 0.66 ms for nine calls; a draw of k-means++ on 1M x 128: 76 -> 72 us. The nodes
// of a captured iteration do not: they follow each other within half a microsecond as they are, and
// with programmatic edges 20 iterations of 100,000 x 32, K=64 took 2.02 instead of 1.87 ms.
inline bool overlap_allowed(cudaStream_t s) {
  if (s == nullptr) return true;  // the legacy stream is never captured
  cudaStreamCaptureStatus st = cudaStreamCaptureStatusNone;
  return cudaStreamIsCapturing(s, &st) == cudaSuccess && st == cudaStreamCaptureStatusNone;
}

// launch(kernel, grid, block, shared memory, stream)(arguments); the kernel begins with grid_enter().
template <class... P>
struct Launch {
  void (*kernel)(P...);
  cudaLaunchConfig_t cfg;
  template <class... A>
  cudaError_t operator()(A&&... args) {
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = at;
    cfg.numAttrs = overlap_allowed(cfg.stream) ? 1 : 0;
    return cudaLaunchKernelEx(&cfg, kernel, std::forward<A>(args)...);
  }
};
template <class... P>
Launch<P...> launch(void (*kernel)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t s) {
  Launch<P...> l;
  l.kernel = kernel;
  l.cfg = cudaLaunchConfig_t{};
  l.cfg.gridDim = grid;
  l.cfg.blockDim = block;
  l.cfg.dynamicSmemBytes = smem;
  l.cfg.stream = s;
  return l;
}

}  // namespace kmgb

#define KMGB_CUDA_TRY(expr)                        \
  do {                                             \
    cudaError_t _e = (expr);                       \
    if (_e != cudaSuccess) return _e;              \
  } while (0)
