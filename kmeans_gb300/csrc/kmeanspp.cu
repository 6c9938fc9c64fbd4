// k-means++ initialisation (the reference declares initAlgorithm and numRetries,
// main/cpp/kmeans.hpp:94-95, kmeans.cpp:29, but implements only its shuffle-and-pick init).
//
// Centers are drawn one at a time, each with probability proportional to D^2, the squared
// distance of a point to its nearest already-chosen center. The draws are reproducible bit for
// bit on the data type T (float or double):
//   * D^2 is computed in T: lane l of a warp accumulates dimensions l, l+32, ... with
//     fma((x-c), (x-c), s) in increasing order, then an xor butterfly over the 32 lanes
//     (s += shfl_xor(s, o), o = 16, 8, 4, 2, 1; every lane ends with the same sum);
//     D^2 = fmin(D^2, distance to the newest center).
//   * The sampling weight of a point is q = uint32 truncation (saturating, NaN -> 0) of
//     D^2 * (2^31 / M) in T, M the largest D^2 after the update (so q <= 2^31). Sums of q are
//     exact 64-bit integers: the order of the parallel sums does not matter.
//   * Draw r takes u = splitmix64(splitmix64(seed) + r) >> 11 (53 bits) and picks the point whose
//     interval [prefix, prefix + q) of the running sum of q holds (u * total) >> 53 (128-bit
//     product). Draw 0, and any draw whose total weight is 0, picks point (u * n) >> 53.
// Per draw: one pass over X (D^2 update and maximum) and one over D^2 (weights and their sums per
// 1024 points; the last block to finish scans the block sums, draws and picks). D^2 is n elements
// of T; reading X bounds the whole initialisation by HBM, so rows whose D^2 a new center cannot lower
// are not read where that can be told (kpp_update_bulk_kernel).
#include "common.cuh"
#include "kernels.h"

namespace kmgb {
namespace {

constexpr int KPP_BLOCK = 1024;  // points per weight-sum block (= threads of the pick kernel)
constexpr int KPP_THREADS = 256;

__host__ __device__ inline uint64_t splitmix64(uint64_t x) {
  x += 0x9E3779B97F4A7C15ull;
  x = (x ^ (x >> 30)) * 0xBF58476D1CE4E5B9ull;
  x = (x ^ (x >> 27)) * 0x94D049BB133111EBull;
  return x ^ (x >> 31);
}

__device__ inline uint64_t draw53(uint64_t seed, uint64_t round) {
  return splitmix64(splitmix64(seed) + round) >> 11;
}

__device__ __forceinline__ float kpp_fma(float a, float b, float c) { return __fmaf_rn(a, b, c); }
__device__ __forceinline__ double kpp_fma(double a, double b, double c) { return __fma_rn(a, b, c); }

// Largest D^2 as an order-preserving unsigned key (D^2 >= 0 or NaN; NaN never raises it).
__device__ __forceinline__ unsigned long long kpp_key(float v) { return __float_as_uint(v); }
__device__ __forceinline__ unsigned long long kpp_key(double v) {
  return (unsigned long long)__double_as_longlong(v);
}
template <typename T>
__device__ __forceinline__ T kpp_unkey(unsigned long long k);
template <>
__device__ __forceinline__ float kpp_unkey<float>(unsigned long long k) {
  return __uint_as_float((unsigned int)k);
}
template <>
__device__ __forceinline__ double kpp_unkey<double>(unsigned long long k) {
  return __longlong_as_double((long long)k);
}

template <typename T>
__device__ __forceinline__ T kpp_scale(unsigned long long mkey) {
  const T m = kpp_unkey<T>(mkey);
  return m > T(0) ? T(2147483648.0) / m : T(0);  // IEEE division in T
}

// Saturating truncation to uint32 (cvt.rzi.u32: NaN and negatives -> 0).
__device__ __forceinline__ unsigned int kpp_weight(float v, float scale) {
  return __float2uint_rz(__fmul_rn(v, scale));
}
__device__ __forceinline__ unsigned int kpp_weight(double v, double scale) {
  return __double2uint_rz(__dmul_rn(v, scale));
}

// Exclusive scan of one value per thread over a 1024-thread block; *total gets the sum.
__device__ unsigned long long block_exclusive_scan(unsigned long long v, unsigned long long* warp_sh,
                                                   unsigned long long* total_sh) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  unsigned long long incl = v;
  for (int o = 1; o < 32; o <<= 1) {
    const unsigned long long t = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= o) incl += t;
  }
  if (lane == 31) warp_sh[warp] = incl;
  __syncthreads();
  if (warp == 0) {
    const unsigned long long w = warp_sh[lane];
    unsigned long long wi = w;
    for (int o = 1; o < 32; o <<= 1) {
      const unsigned long long t = __shfl_up_sync(0xffffffffu, wi, o);
      if (lane >= o) wi += t;
    }
    warp_sh[lane] = wi - w;
    if (lane == 31) *total_sh = wi;
  }
  __syncthreads();
  const unsigned long long r = warp_sh[warp] + incl - v;
  __syncthreads();  // warp_sh may be reused by the caller's next scan
  return r;
}

// D^2 of the points of one 1024-point block against the newest center (row *pick); the block's
// largest D^2 raises *max_key. A warp takes KPP_ROWS rows at a time, their loads interleaved so
// that each lane keeps 4 x KPP_ROWS loads in flight; every row keeps its own lane-partial fma
// chain in increasing dimension order, so the sums are those of one row at a time.
constexpr int KPP_ROWS = 4;

template <typename T>
__global__ void __launch_bounds__(KPP_THREADS)
kpp_update_kernel(const T* X, long long ldx, long long n, int d,
                  const int* pick, T* __restrict__ d2, int first,
                  unsigned long long* __restrict__ max_key) {
  if (grid_enter()) return;
  __shared__ unsigned long long wmax[KPP_THREADS / 32];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const T* c = X + (size_t)(*pick) * ldx;
  T mx = T(0);
  const long long p0 = (long long)blockIdx.x * KPP_BLOCK;
  const long long pend = min(n, p0 + KPP_BLOCK);
  for (long long pr = p0 + (long long)warp * KPP_ROWS; pr < pend;
       pr += (long long)(KPP_THREADS / 32) * KPP_ROWS) {
    const T* x[KPP_ROWS];
    T s[KPP_ROWS];
#pragma unroll
    for (int r = 0; r < KPP_ROWS; ++r) {
      // rows past the end re-read the last valid row (never stored)
      x[r] = X + (size_t)min(pr + r, pend - 1) * ldx;
      s[r] = T(0);
    }
#pragma unroll 4
    for (int t = lane; t < d; t += 32) {
      const T cv = ld(c + t);
#pragma unroll
      for (int r = 0; r < KPP_ROWS; ++r) {
        const T u = ld(x[r] + t) - cv;
        s[r] = kpp_fma(u, u, s[r]);
      }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
#pragma unroll
      for (int r = 0; r < KPP_ROWS; ++r) s[r] = s[r] + __shfl_xor_sync(0xffffffffu, s[r], o);
    }
#pragma unroll
    for (int r = 0; r < KPP_ROWS; ++r) {
      const long long pt = pr + r;
      if (pt < pend) {
        const T v = first ? s[r] : fmin(d2[pt], s[r]);
        if (lane == 0) d2[pt] = v;
        mx = fmax(mx, v);
      }
    }
  }
  if (lane == 0) wmax[warp] = kpp_key(mx);
  __syncthreads();
  if (threadIdx.x == 0) {
    unsigned long long m = 0;
    for (int w = 0; w < KPP_THREADS / 32; ++w) m = max(m, wmax[w]);
    atomicMax(max_key, m);
  }
}

// The same D^2 update with X staged through shared memory: a producer warp streams chunks of
// `rows_per_stage` contiguous rows (and their old D^2 values) with cp.async.bulk into a ring of
// `stages` buffers, so the bytes in flight per SM are the ring's, not the registers'; 8
// consumer warps compute each row exactly as kpp_update_kernel does (lane l: dims l, l+32, ...
// from shared memory, fma chain, xor butterfly). Needs 16-byte aligned rows (ldx * sizeof(T) a
// multiple of 16, X 16-byte aligned) and d2 padded to a multiple of 4 rows. Every wait is
// bounded; on a timeout the CTA records KMGB_DEV_TIMEOUT_FULL/EMPTY in *err, waits (bounded)
// for its copies in flight and returns.
constexpr int KPP_CONSUMERS = 8;
constexpr int KPP_BULK_THREADS = (KPP_CONSUMERS + 1) * 32;
constexpr int KPP_MAX_STAGES = 8;

__device__ __forceinline__ void bulk_g2s(uint32_t dst, const void* src, uint32_t bytes,
                                         uint32_t bar) {
  asm volatile(
      "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
          dst),
      "l"(reinterpret_cast<uint64_t>(src)), "r"(bytes), "r"(bar)
      : "memory");
}

//
// Rows that need not be read (KppNear, from draw 2 on): near[i] is the draw whose center gave D^2_i,
// and cc[q] a lower bound of the squared distance from draw q's center to the new one. Where
// cc[near[i]] >= 4 D^2_i (1 + slack), the triangle inequality puts the row at least as far from the new
// center as from its own, by more than the rounding of both computed distances, so the minimum is
// D^2_i again, bit for bit. A warp tests 32 rows at a time and gathers the others, eight rows'
// loads in flight; each row's sum is formed as above. The share of rows read falls with the draws
// where clusters lie apart. At 1M x 128 a draw streams every row in 83 us (96 us before the eight-row
// reduction below: the consumers' shuffles held the ring back) and gathers every row in 103 us, so a
// draw gathers only when the last gathering draw read at most kKppGatherShare of the rows, and every
// 16th draw gathers to look again. 256 draws from 256 Gaussians: 28.3 ms reading every row, 19.4 ms so.
constexpr double kKppGatherShare = 0.7;

struct KppNear {
  int* near;               // [n] draw of the nearest center; null: every row is read
  const void* cc;          // [draw] lower bounds (T) of squared distances to the new center
  unsigned int* active;    // rows read by the last gathering draw, [1] its running count
  int draw;
};

template <typename T>
__device__ __forceinline__ bool kpp_in_range(T v);
template <>
__device__ __forceinline__ bool kpp_in_range<float>(float v) { return v >= 1e-30f && v < 1e37f; }
template <>
__device__ __forceinline__ bool kpp_in_range<double>(double v) { return v >= 1e-290 && v < 1e300; }

// Relative error of a computed squared distance: at most d / 32 + 7 roundings, the difference's twice.
template <typename T>
__device__ __forceinline__ T kpp_rel(int d) {
  return (T)(d / 32 + 16) * (sizeof(T) == 4 ? (T)5.9604645e-8 : (T)1.1102230246251565e-16);
}

// Eight rows' lane partials to their butterfly sums: lanes 4r .. 4r+3 end with row r's. The first three
// steps of the butterfly halve the rows a lane still carries, nine shuffles for the eight rows instead
// of forty; every addition joins the same two partials (in either order), so the sums are
// those of a full butterfly, bit for bit.
template <typename T>
__device__ __forceinline__ T kpp_reduce8(T (&s)[8], int lane) {
#pragma unroll
  for (int h = 4; h > 0; h >>= 1) {
    const int o = 4 * h;
    const bool up = lane & o;
#pragma unroll
    for (int r = 0; r < h; ++r) {
      const T keep = up ? s[r + h] : s[r], send = up ? s[r] : s[r + h];
      s[r] = keep + __shfl_xor_sync(0xffffffffu, send, o);
    }
  }
  s[0] = s[0] + __shfl_xor_sync(0xffffffffu, s[0], 2);
  s[0] = s[0] + __shfl_xor_sync(0xffffffffu, s[0], 1);
  return s[0];
}

template <typename T>
__device__ __forceinline__ T kpp_gather_rows(const T* __restrict__ X, long long ldx, long long n, int d,
                                             const T* cs, T* __restrict__ d2, const KppNear& nr) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, warps = blockDim.x >> 5;
  const T* cc = static_cast<const T*>(nr.cc);
  const T slack = T(4) * (T(1) + T(16) * kpp_rel<T>(d));
  T mx = T(0);
  unsigned int read = 0;
  const long long step = (long long)gridDim.x * warps * 32;
  long long i0 = ((long long)blockIdx.x * warps + warp) * 32;
  T v = T(0);
  int a = 0;
  if (i0 + lane < n) {
    v = d2[i0 + lane];
    a = nr.near[i0 + lane];
  }
  for (; i0 < n; i0 += step) {
    const long long i = i0 + lane;
    const bool in = i < n;
    const T cur = v;
    const int cura = a;
    if (i + step < n) {  // the next group's values in flight
      v = d2[i + step];
      a = nr.near[i + step];
    }
    const bool skip = !in || cur == T(0) ||
                      (kpp_in_range(cur) && ld(cc + cura) >= slack * cur);
    unsigned todo = __ballot_sync(0xffffffffu, !skip);
    read += __popc(todo);
    if (in && skip) mx = fmax(mx, cur);
    while (todo) {
      int row[8];
#pragma unroll
      for (int r = 0; r < 8; ++r) {
        row[r] = todo ? __ffs(todo) - 1 : -1;
        todo &= todo - 1;
      }
      T sv[8];
      const T* x[8];
      int own = row[0];  // the row whose sum this lane ends with
#pragma unroll
      for (int r = 0; r < 8; ++r) {
        sv[r] = T(0);
        x[r] = X + (size_t)(i0 + (row[r] >= 0 ? row[r] : row[0])) * ldx;
        if ((lane >> 2) == r) own = row[r];
      }
      // 512 bytes of each of the eight rows in flight together (slots without a row re-read a row)
      constexpr int kSteps = 16 / sizeof(T);
      for (int t0 = lane; t0 < d; t0 += 32 * kSteps) {
        T xv[kSteps][8];
#pragma unroll
        for (int q = 0; q < kSteps; ++q)
#pragma unroll
          for (int r = 0; r < 8; ++r) xv[q][r] = t0 + 32 * q < d ? ld(x[r] + t0 + 32 * q) : T(0);
#pragma unroll
        for (int q = 0; q < kSteps; ++q) {
          if (t0 + 32 * q >= d) break;
          const T cv = cs[t0 + 32 * q];
#pragma unroll
          for (int r = 0; r < 8; ++r) {
            const T u = xv[q][r] - cv;
            sv[r] = kpp_fma(u, u, sv[r]);
          }
        }
      }
      const T sum = kpp_reduce8(sv, lane);
      const T old = __shfl_sync(0xffffffffu, cur, own >= 0 ? own : 0);
      if ((lane & 3) == 0 && own >= 0) {
        const T nv = fmin(old, sum);
        if (nv != old && nv == nv) {
          d2[i0 + own] = nv;
          nr.near[i0 + own] = nr.draw;
        }
        mx = fmax(mx, nv);
      }
    }
  }
  // (one more, so that a draw that read nothing still counts as measured)
  if (lane == 0 && blockIdx.x == 0 && warp == 0) ++read;
  if (lane == 0 && read) atomicAdd(nr.active + 1, read);
  for (int o = 16; o > 0; o >>= 1) mx = fmax(mx, __shfl_xor_sync(0xffffffffu, mx, o));
  return mx;
}

template <typename T>
__global__ void __launch_bounds__(KPP_BULK_THREADS)
kpp_update_bulk_kernel(const T* X, long long ldx, long long n, int d,
                       const int* pick, T* __restrict__ d2, int first,
                       unsigned long long* __restrict__ max_key, int rows_per_stage, int stages,
                       int* __restrict__ err, KppNear nr) {
  if (grid_enter()) return;
  extern __shared__ __align__(128) unsigned char kpp_smem[];
  __shared__ __align__(8) uint64_t full_bar[KPP_MAX_STAGES], empty_bar[KPP_MAX_STAGES];
  __shared__ unsigned long long wmax[KPP_CONSUMERS + 1];
  __shared__ int abort_flag;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const long long row_elems = ldx;
  const uint32_t row_bytes = (uint32_t)(ldx * (long long)sizeof(T));
  const uint32_t xstage_bytes = row_bytes * (uint32_t)rows_per_stage;
  T* cs = reinterpret_cast<T*>(kpp_smem);                              // the new center
  unsigned char* ring = kpp_smem + ((d * sizeof(T) + 127) / 128) * 128;  // X stages, then D^2
  T* dring = reinterpret_cast<T*>(ring + (size_t)stages * xstage_bytes);
  const long long nchunks = (n + rows_per_stage - 1) / rows_per_stage;

  const T* c = X + (size_t)(*pick) * ldx;
  for (int t = threadIdx.x; t < d; t += blockDim.x) cs[t] = c[t];
  if (threadIdx.x == 0) {
    abort_flag = 0;
    for (int i = 0; i < stages; ++i) {
      mbar_init(smem_u32(&full_bar[i]), 1);
      mbar_init(smem_u32(&empty_bar[i]), KPP_CONSUMERS);
    }
    fence_mbar_init();
  }
  __syncthreads();
  // the last gathering draw's count is final: it was written by an earlier launch
  const bool gather = nr.near && !first &&
                      (nr.draw % 16 == 0 ||
                       (double)nr.active[0] <= kKppGatherShare * (double)n);

  if (gather) {
    const T m = kpp_gather_rows<T>(X, ldx, n, d, cs, d2, nr);
    if (lane == 0) wmax[warp] = kpp_key(m);
  } else if (warp == KPP_CONSUMERS) {  // producer
    if (lane == 0) {
      long long it = 0;
      for (long long ch = blockIdx.x; ch < nchunks; ch += gridDim.x, ++it) {
        const int sidx = (int)(it % stages);
        if (it >= stages &&
            !mbar_wait(smem_u32(&empty_bar[sidx]), (uint32_t)(((it / stages) - 1) & 1),
                       &abort_flag, err, KMGB_DEV_TIMEOUT_EMPTY))
          break;
        const long long r0 = ch * rows_per_stage;
        const int rows = (int)min((long long)rows_per_stage, n - r0);
        const uint32_t xb = row_bytes * (uint32_t)rows;
        // D^2 slice rounded up to 16 bytes (d2 holds a multiple of 4 rows)
        const uint32_t db = first ? 0u : (uint32_t)((((rows + 3) & ~3)) * sizeof(T));
        const uint32_t bar = smem_u32(&full_bar[sidx]);
        mbar_arrive_expect_tx(bar, xb + db);
        bulk_g2s(smem_u32(ring + (size_t)sidx * xstage_bytes), X + (size_t)r0 * row_elems, xb, bar);
        if (db) bulk_g2s(smem_u32(dring + (size_t)sidx * rows_per_stage), d2 + r0, db, bar);
      }
      // copies still in flight (only after an abort) must land before the CTA exits
      const long long issued = it;
      for (long long j = issued - 1; j >= 0 && j >= issued - stages; --j) {
        const uint32_t bar = smem_u32(&full_bar[j % stages]);
        const uint32_t par = (uint32_t)((j / stages) & 1);
        const long long t0 = clock64();
        while (!mbar_try_wait(bar, par) &&
               (unsigned long long)(clock64() - t0) < KMGB_WAIT_CYCLES) {
        }
      }
    }
    __syncwarp();
  } else {  // consumers
    T mx = T(0);
    long long it = 0;
    for (long long ch = blockIdx.x; ch < nchunks; ch += gridDim.x, ++it) {
      const int sidx = (int)(it % stages);
      if (!mbar_wait(smem_u32(&full_bar[sidx]), (uint32_t)((it / stages) & 1), &abort_flag, err,
                     KMGB_DEV_TIMEOUT_FULL))
        break;
      const long long r0 = ch * rows_per_stage;
      const int rows = (int)min((long long)rows_per_stage, n - r0);
      const T* xs = reinterpret_cast<const T*>(ring + (size_t)sidx * xstage_bytes);
      const T* ds = dring + (size_t)sidx * rows_per_stage;
      for (int g = warp * 8; g < rows; g += KPP_CONSUMERS * 8) {
        T sv[8];
        const T* xr[8];
#pragma unroll
        for (int r = 0; r < 8; ++r) {
          sv[r] = T(0);
          xr[r] = xs + (size_t)min(g + r, rows - 1) * row_elems;
        }
#pragma unroll 4
        for (int t = lane; t < d; t += 32) {
          const T cv = cs[t];
#pragma unroll
          for (int r = 0; r < 8; ++r) {
            const T u = xr[r][t] - cv;
            sv[r] = kpp_fma(u, u, sv[r]);
          }
        }
        const T sum = kpp_reduce8(sv, lane);
        const int row = g + (lane >> 2);
        if ((lane & 3) == 0 && row < rows) {
          const T old = first ? sum : ds[row];
          const T v = first ? sum : fmin(old, sum);
          d2[r0 + row] = v;
          if (nr.near && (first || v != old)) nr.near[r0 + row] = first ? 0 : nr.draw;
          mx = fmax(mx, v);
        }
      }
      __syncwarp();
      if (lane == 0) mbar_arrive(smem_u32(&empty_bar[sidx]));
    }
    for (int o = 16; o > 0; o >>= 1) mx = fmax(mx, __shfl_xor_sync(0xffffffffu, mx, o));
    if (lane == 0) wmax[warp] = kpp_key(mx);
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    unsigned long long m = 0;
    for (int w = 0; w < KPP_CONSUMERS + (gather ? 1 : 0); ++w) m = max(m, wmax[w]);
    atomicMax(max_key, m);
  }
}

// Lower bounds of the squared distances from the newest center (row *pick) to the centers of draws
// 0 .. draw-1 (rows picks[q]), one warp each; block 0 closes the last gathering draw's count.
template <typename T>
__global__ void kpp_center_dist_kernel(const T* X, long long ldx, int d,
                                       const int* picks, int draw, T* __restrict__ cc,
                                       unsigned int* __restrict__ active) {
  if (grid_enter()) return;
  const int q = (int)((blockIdx.x * blockDim.x + threadIdx.x) >> 5);
  const int lane = threadIdx.x & 31;
  if (q == 0 && lane == 0 && active[1]) {
    active[0] = active[1];
    active[1] = 0;
  }
  if (q >= draw) return;
  const T* c = X + (size_t)picks[draw] * ldx;
  const T* o = X + (size_t)picks[q] * ldx;
  T s = T(0);
  for (int t = lane; t < d; t += 32) {
    const T u = ld(c + t) - ld(o + t);
    s = kpp_fma(u, u, s);
  }
  for (int m = 16; m > 0; m >>= 1) s = s + __shfl_xor_sync(0xffffffffu, s, m);
  if (lane == 0) cc[q] = s * (T(1) - T(4) * kpp_rel<T>(d));
}

// The draw of round `round`. Every block adds the weights q of its 1024-point blocks (exact sums); the
// last block to finish scans them, draws, finds the 1024-point block holding the target, then the
// point inside it (1024 threads, one point each), and writes *pick and picks[round]. Without weights
// (round 0) the sums are zero and the draw uniform.
template <typename T>
__global__ void __launch_bounds__(KPP_BLOCK)
kpp_draw_kernel(long long n, const T* d2, unsigned long long* blocksum, long long nblocks,
                bool weights, const unsigned long long* max_key,
                unsigned long long* __restrict__ next_max_key, unsigned int* ticket,
                unsigned long long seed, int round, int* __restrict__ pick, int* __restrict__ picks) {
  if (grid_enter()) return;
  __shared__ unsigned long long warp_sh[32];
  __shared__ unsigned long long total_sh, off_sh, tot2_sh;
  __shared__ long long block_sh, chosen_sh;
  __shared__ bool last_sh;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const T scale = weights ? kpp_scale<T>(*max_key) : T(0);
  if (weights) {  // one warp per 1024-point block, its loads in flight together
    for (long long b = blockIdx.x * 32LL + warp; b < nblocks; b += gridDim.x * 32LL) {
      const long long p0 = b * (long long)KPP_BLOCK + lane;
      T v[KPP_BLOCK / 32];
#pragma unroll
      for (int i = 0; i < KPP_BLOCK / 32; ++i) v[i] = p0 + 32 * i < n ? ld(d2 + p0 + 32 * i) : T(0);
      unsigned long long q = 0;
#pragma unroll
      for (int i = 0; i < KPP_BLOCK / 32; ++i) q += kpp_weight(v[i], scale);
      for (int o = 16; o > 0; o >>= 1) q += __shfl_xor_sync(0xffffffffu, q, o);
      if (lane == 0) __stcg(blocksum + b, q);
    }
    __syncthreads();
  }
  if (tid == 0) {
    __threadfence();  // this block's sums before its ticket
    last_sh = atomicAdd(ticket, 1u) == gridDim.x - 1;
    block_sh = -1;
    chosen_sh = -1;
  }
  __syncthreads();
  if (!last_sh) return;
  __threadfence();
  if (tid == 0) *ticket = 0;
  // each thread sums a contiguous run of blocks
  const long long per = (nblocks + KPP_BLOCK - 1) / KPP_BLOCK;
  const long long b0 = (long long)tid * per, b1 = min(nblocks, b0 + per);
  unsigned long long s = 0;
  for (long long b = b0; b < b1; ++b) s += weights ? __ldcg(blocksum + b) : 0ull;
  unsigned long long off = block_exclusive_scan(s, warp_sh, &total_sh);
  const unsigned long long total = total_sh;
  const uint64_t u = draw53(seed, (uint64_t)round);
  const unsigned long long uniform = __umul64hi(u << 11, (unsigned long long)n);  // (u*n) >> 53
  if (tid == 0) *next_max_key = 0;  // the next draw's maximum (not read by this draw)
  if (total == 0) {
    if (tid == 0) {
      *pick = (int)uniform;
      picks[round] = (int)uniform;
    }
    return;
  }
  const unsigned long long target = __umul64hi(u << 11, total);  // (u * total) >> 53 < total
  if (off <= target && target < off + s) {  // exactly one thread's run holds the target
    for (long long b = b0; b < b1; ++b) {
      const unsigned long long nx = off + __ldcg(blocksum + b);
      if (nx > target) {
        block_sh = b;
        off_sh = off;
        break;
      }
      off = nx;
    }
  }
  __syncthreads();
  const long long b = block_sh;  // >= 0: the runs partition [0, total)
  const long long pt = b * (long long)KPP_BLOCK + tid;
  const unsigned long long q = (b >= 0 && pt < n) ? kpp_weight(d2[pt], scale) : 0ull;
  const unsigned long long ex = off_sh + block_exclusive_scan(q, warp_sh, &tot2_sh);
  if (q > 0 && ex <= target && target < ex + q) chosen_sh = pt;
  __syncthreads();
  if (tid == 0) {
    const long long c = chosen_sh >= 0 ? chosen_sh : (long long)uniform;
    *pick = (int)c;
    picks[round] = (int)c;
  }
}

template <typename T>
__global__ void kpp_gather_kernel(const T* X, long long ldx, int d,
                                  const int* picks, int k, T* __restrict__ C,
                                  long long ldc) {
  if (grid_enter()) return;
  for (long long e = (long long)blockIdx.x * blockDim.x + threadIdx.x; e < (long long)k * d;
       e += (long long)gridDim.x * blockDim.x) {
    const int j = (int)(e / d), t = (int)(e - (long long)j * d);
    C[(size_t)j * ldc + t] = X[(size_t)picks[j] * ldx + t];
  }
}

// Ring geometry of kpp_update_bulk_kernel for rows of `row_bytes`: rows per stage (a multiple of 8, a
// warp's step, about 32 KB of rows, whole rounds of the 8 consumer warps where more than one; 4 very
// wide ones) and stages (2..8) within a shared-memory budget that leaves room for two CTAs per SM.
// Returns false when the rows are too wide (the register kernel is used then).
constexpr size_t KPP_SMEM_BUDGET = 100 * 1024;

bool kpp_bulk_plan(long long row_bytes, int elem, int d, int* rows_per_stage, int* stages,
                   size_t* smem) {
  long long rps = (32768 / row_bytes) & ~7LL;
  if (rps < 8) rps = 8;
  if (rps > 64 && rps % 64) rps -= rps % 64;
  const long long center = ((long long)d * elem + 127) / 128 * 128;
  if (2 * rps * (row_bytes + elem) + center > (long long)KPP_SMEM_BUDGET) rps = 4;
  const long long per_stage = rps * row_bytes + rps * elem;
  long long st = ((long long)KPP_SMEM_BUDGET - center) / per_stage;
  if (st > KPP_MAX_STAGES) st = KPP_MAX_STAGES;
  if (st < 2) return false;
  *rows_per_stage = (int)rps;
  *stages = (int)st;
  *smem = (size_t)(center + st * per_stage);
  return true;
}

// Rows are skipped only where reading X costs more than the launch that prepares the test: from the
// size of the L2 on, a draw's pass takes 24 us or more.
constexpr long long KPP_NEAR_MIN_BYTES = 128LL << 20;

template <typename T>
cudaError_t kmeanspp_impl(const T* X, long long ldx, long long n, int d, int k,
                          unsigned long long seed, T* C, long long ldc, int* picks, const KppWork<T>& w,
                          int* err, cudaStream_t s) {
  if (n <= 0 || d <= 0 || k <= 0 || k > n || n > 0x7fffffffLL || ldx < d || ldc < d)
    return cudaErrorInvalidValue;
  const long long nb = (n + KPP_BLOCK - 1) / KPP_BLOCK;
  const long long row_bytes = ldx * (long long)sizeof(T);
  int rps = 0, stages = 0;
  size_t smem = 0;
  const bool bulk = (row_bytes % 16) == 0 && (reinterpret_cast<uintptr_t>(X) % 16) == 0 &&
                    (reinterpret_cast<uintptr_t>(w.d2) % 16) == 0 &&
                    kpp_bulk_plan(row_bytes, (int)sizeof(T), d, &rps, &stages, &smem);
  int grid = 0;
  if (bulk) {
    KMGB_CUDA_TRY(cudaFuncSetAttribute(kpp_update_bulk_kernel<T>,
                                       cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       (int)KPP_SMEM_BUDGET));
    int per_sm = 0;
    KMGB_CUDA_TRY(cudaOccupancyMaxActiveBlocksPerMultiprocessor(
        &per_sm, kpp_update_bulk_kernel<T>, KPP_BULK_THREADS, smem));
    const long long chunks = (n + rps - 1) / rps;
    grid = (int)min((long long)kmgb::num_sms() * max(per_sm, 1), chunks);
  }
  // scalars: [0], [1] the maxima of alternate draws (draw r clears draw r+1's), [2] the newest
  // center's row, [3] the draw's block ticket, [4] rows read by the last gathering draw and the
  // running count (all ones: none yet)
  unsigned long long* mx = w.scalars;
  int* pick = reinterpret_cast<int*>(w.scalars + 2);
  unsigned int* ticket = reinterpret_cast<unsigned int*>(w.scalars + 3);
  KppNear nr{};
  if (bulk && w.near && w.cc && n * row_bytes >= KPP_NEAR_MIN_BYTES) {
    nr.near = w.near;
    nr.cc = w.cc;
    nr.active = reinterpret_cast<unsigned int*>(w.scalars + 4);
    KMGB_CUDA_TRY(cudaMemsetAsync(nr.active, 0xff, sizeof(unsigned int), s));
    KMGB_CUDA_TRY(cudaMemsetAsync(nr.active + 1, 0, sizeof(unsigned int), s));
  }
  KMGB_CUDA_TRY(cudaMemsetAsync(mx, 0, 4 * sizeof(unsigned long long), s));
  const long long dblocks = (nb + 31) / 32, most = kmgb::num_sms();  // a warp per 1024 points
  const unsigned dgrid = (unsigned)(dblocks < most ? dblocks : most);
  // draw 0: zero total weight, so uniform
  launch(kpp_draw_kernel<T>, 1, KPP_BLOCK, 0, s)(n, w.d2, w.blocksum, nb, false, mx, mx + 1, ticket, seed, 0,
                                             pick, picks);
  count_launches(1);
  for (int r = 1; r < k; ++r) {
    unsigned long long* m = mx + (r & 1);
    nr.draw = r - 1;
    if (nr.near && r > 1) {
      launch(kpp_center_dist_kernel<T>, (unsigned)((nr.draw + 7) / 8), 256, 0, s)(
          X, ldx, d, picks, nr.draw, static_cast<T*>(w.cc), nr.active);
      count_launches(1);
    }
    if (bulk)
      launch(kpp_update_bulk_kernel<T>, grid, KPP_BULK_THREADS, smem, s)(
          X, ldx, n, d, pick, w.d2, r == 1, m, rps, stages, err, nr);
    else
      launch(kpp_update_kernel<T>, (unsigned)nb, KPP_THREADS, 0, s)(X, ldx, n, d, pick, w.d2, r == 1, m);
    launch(kpp_draw_kernel<T>, dgrid, KPP_BLOCK, 0, s)(n, w.d2, w.blocksum, nb, true, m,
                                                   mx + ((r + 1) & 1), ticket, seed, r, pick, picks);
    count_launches(2);
  }
  launch(kpp_gather_kernel<T>, kmgb::num_sms() * 4, 256, 0, s)(X, ldx, d, picks, k, C, ldc);
  count_launches(1);
  return cudaGetLastError();
}

}  // namespace

long long kmeanspp_blocks(long long n) { return (n + KPP_BLOCK - 1) / KPP_BLOCK; }
long long kmeanspp_d2_elems(long long n) { return (n + 3) / 4 * 4; }

cudaError_t launch_kmeanspp(const float* X, long long ldx, long long n, int d, int k,
                            unsigned long long seed, float* C, long long ldc, int* picks,
                            const KppWork<float>& w, int* err, cudaStream_t s) {
  return kmeanspp_impl<float>(X, ldx, n, d, k, seed, C, ldc, picks, w, err, s);
}

cudaError_t launch_kmeanspp(const double* X, long long ldx, long long n, int d, int k,
                            unsigned long long seed, double* C, long long ldc, int* picks,
                            const KppWork<double>& w, int* err, cudaStream_t s) {
  return kmeanspp_impl<double>(X, ldx, n, d, k, seed, C, ldc, picks, w, err, s);
}

}  // namespace kmgb
