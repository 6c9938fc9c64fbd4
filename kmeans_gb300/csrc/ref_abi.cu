// The reference's per-kernel C entry points (main/cuda/KmeansCudaKernels.h:198-474) on the GB300
// kernels. Same names, argument meaning and kmeansCudaErrorStatus codes; asynchronous on the
// default stream like the reference; the reference's scratch arguments (Bpadded, C, Cindices,
// normRowsOfA_squared in ClosestCenters) are accepted and not needed. Temporary buffers are
// stream-ordered on the default stream: cudaMallocAsync, and for ClosestCenters one allocation from
// the library's pool for calls (devmem.cu).
#include <algorithm>
#include <cfloat>
#include <cmath>

#include "../../include/kmeans_gb300.h"
#include "common.cuh"
#include "kernels.h"

using namespace kmgb;

namespace {

const cudaStream_t kDefault = 0;

template <typename T>
cudaError_t tmp_alloc(T** p, size_t count) {
  return cudaMallocAsync(reinterpret_cast<void**>(p), sizeof(T) * (count ? count : 1), kDefault);
}
void tmp_free(void* p) {
  if (p) cudaFreeAsync(p, kDefault);
}

__global__ void copy_pad_kernel(const float* A, long long m, int d, float* __restrict__ Ap,
                                long long ld) {
  if (grid_enter()) return;
  const long long total = m * ld;
  for (long long e = (long long)blockIdx.x * blockDim.x + threadIdx.x; e < total;
       e += (long long)gridDim.x * blockDim.x) {
    const long long r = e / ld;
    const int c = (int)(e % ld);
    Ap[e] = c < d ? A[(size_t)r * d + c] : 0.0f;
  }
}

// FP64 arg-min of nb_j - 2 A_i.B_j (B is d x k, K fastest); one warp per row, lanes over j. list
// (nullable): only the rows list[0 .. *count), or every row where *redo is set.
__global__ void closest_fp64_kernel(int m0, int m, int d, const double* A, int k,
                                    const double* B, const double* nb,
                                    int* __restrict__ out, const int* list,
                                    const int* count, const int* redo) {
  if (grid_enter()) return;
  if (list && pinned(redo) != 0) list = nullptr;
  extern __shared__ double xs_all[];
  const int warps = blockDim.x >> 5, w = threadIdx.x >> 5, lane = threadIdx.x & 31;
  double* xs = xs_all + (size_t)w * d;
  const long long todo = list ? (long long)*count : m;
  for (long long slot = (long long)blockIdx.x * warps + w; slot < todo;
       slot += (long long)gridDim.x * warps) {
    const long long i = list ? (long long)list[slot] : slot;
    for (int t = lane; t < d; t += 32) xs[t] = A[(size_t)i * d + t];
    __syncwarp();
    double best = INFINITY;
    int bi = -1;
    for (int j = lane; j < k; j += 32) {
      double s = 0.0;
      for (int t = 0; t < d; ++t) s = fma(xs[t], B[(size_t)t * k + j], s);
      const double v = fma(-2.0, s, nb[j]);
      if (v < best) {
        best = v;
        bi = j;
      }
    }
    for (int o = 16; o > 0; o >>= 1) {
      const double ob = __shfl_xor_sync(0xffffffffu, best, o);
      const int oi = __shfl_xor_sync(0xffffffffu, bi, o);
      const bool take = (ob < best) || (ob == best && (unsigned)oi < (unsigned)bi);
      best = take ? ob : best;
      bi = take ? oi : bi;
    }
    if (lane == 0) out[m0 + i] = bi < 0 ? 0 : bi;
    __syncwarp();
  }
}

// rowTransformMinimum with the reference's expression (RowTransformMinimum.cu:27-50).
template <typename T>
__global__ void row_transform_min_kernel(int m0, int m, int n, const T* na,
                                         const T* nbv, const T* in,
                                         int* __restrict__ out) {
  if (grid_enter()) return;
  const int warps = blockDim.x >> 5, w = threadIdx.x >> 5, lane = threadIdx.x & 31;
  for (long long i = (long long)blockIdx.x * warps + w; i < m; i += (long long)gridDim.x * warps) {
    T best = (T)FLT_MAX;
    int bi = -1;
    const T a = na[i];
    for (int j = lane; j < n; j += 32) {
      T v;
      if (sizeof(T) == 4) {
        const float s = (float)a + (float)nbv[j];
        v = (T)(float)((double)s - 2.0 * (double)in[(size_t)i * n + j]);
      } else {
        v = a + nbv[j] - (T)2.0 * in[(size_t)i * n + j];
      }
      if (v < best) {
        best = v;
        bi = j;
      }
    }
    for (int o = 16; o > 0; o >>= 1) {
      const T ob = __shfl_xor_sync(0xffffffffu, best, o);
      const int oi = __shfl_xor_sync(0xffffffffu, bi, o);
      const bool take = (ob < best) || (ob == best && (unsigned)oi < (unsigned)bi);
      best = take ? ob : best;
      bi = take ? oi : bi;
    }
    if (lane == 0) out[m0 + i] = bi;
  }
}

__device__ __forceinline__ void ff_two_sum(float a, float b, float& s, float& e) {
  s = __fadd_rn(a, b);
  const float bp = __fsub_rn(s, a);
  e = __fadd_rn(__fsub_rn(a, __fsub_rn(s, bp)), __fsub_rn(b, bp));
}

// Sum over a block's threads (256), for thread 0.
__device__ __forceinline__ double block_sum(double acc) {
  __shared__ double red[8];
  for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = acc;
  __syncthreads();
  double t = 0.0;
  if (threadIdx.x == 0)
    for (int i = 0; i < 8; ++i) t += red[i];
  return t;
}

// Squared distances of the rows to their centers, block partial sums. Bound by HBM (every row once;
// the centers come from L1/L2), with FP32 data also by GB300's narrow FP64 pipe as long as every
// element is widened (898,790 x 128: 1.21 ms): there the terms run on the FP32 pipe as error-free
// float-float values -- u = x - c exactly (TwoSum), u^2 = p + e (FMA), TwoSum accumulation -- and a
// lane widens a pair at every kSegTerms terms: the low part is a plain sum, so its rounding errors, 2^-24
// of it each, stay within 2^-35 of the pair (some 2^-44 as they fall), however wide the rows. A segment of
// kSegSteps rows in which a pair leaves the range where that holds (overflow, squares near the subnormals,
// NaN) is evaluated in FP64.
// L lanes share a row, 16 bytes each at a time where rows are aligned; four rows and the next four's
// labels are in flight without a branch per row (898,790 x 128: 155 -> 129 us, at some two thirds of the
// issue slots).
constexpr int kSegSteps = 32, kSegTerms = 128;

template <int L>
__global__ void __launch_bounds__(256)
compactness_ff_kernel(long long m, int n, const float* data, const int* idx,
                      const float* centers, bool vec, double* __restrict__ partial) {
  if (grid_enter()) return;
  constexpr int G = 32 / L;
  const int lane = threadIdx.x & 31, grp = lane / L, sub = lane % L;
  const long long w0 = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const long long nw = ((long long)gridDim.x * blockDim.x) >> 5;
  double acc = 0.0;
  for (long long s0 = w0 * G * kSegSteps; s0 < m; s0 += nw * G * kSegSteps) {
    float hi = 0.0f, lo = 0.0f, mx = 0.0f;
    double seg = 0.0;
    bool off = false;
    int terms = 0;
    auto widen = [&] {
      off |= !(hi < 1e37f && (hi > 1e-24f || mx == 0.0f));
      seg += (double)hi + (double)lo;
      hi = lo = mx = 0.0f;
      terms = 0;
    };
    auto term = [&](float x, float c) {
      float uh, ul, t, err;
      ff_two_sum(x, -c, uh, ul);
      const float p = __fmul_rn(uh, uh);
      const float e = __fmaf_rn(uh, uh, -p);
      const float r = __fmaf_rn(ul, ul, __fmaf_rn(__fadd_rn(uh, uh), ul, e));
      ff_two_sum(hi, p, t, err);
      hi = t;
      lo = __fadd_rn(lo, __fadd_rn(err, r));
      mx = fmaxf(mx, fabsf(uh));
    };
    // U rows at a time, the next ones' labels with this batch's elements; rows past the end and
    // dimensions past n add zeros, which change neither hi nor lo
    constexpr int U = 4;
    int id[U], nx[U];
    auto load_ids = [&](int i, int (&o)[U]) {
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const long long r = s0 + (i + u) * G + grp;
        o[u] = i < kSegSteps && r < m ? ld(idx + r) : -1;
      }
    };
    load_ids(0, id);
    for (int i = 0; i < kSegSteps; i += U) {
      load_ids(i + U, nx);
      if (vec) {
        for (int t0 = 0; t0 < n; t0 += 4 * L) {
          const int t = t0 + 4 * sub < n ? t0 + 4 * sub : 0;
          float4 xv[U], cv[U];
#pragma unroll
          for (int u = 0; u < U; ++u) {
            const long long r = s0 + (i + u) * G + grp;
            xv[u] = ld(reinterpret_cast<const float4*>(data + (size_t)(id[u] >= 0 ? r : 0) * n + t));
            cv[u] = ld(reinterpret_cast<const float4*>(centers + (size_t)max(id[u], 0) * n + t));
          }
#pragma unroll
          for (int u = 0; u < U; ++u) {
            if (id[u] < 0 || t0 + 4 * sub >= n) xv[u] = cv[u] = make_float4(0.f, 0.f, 0.f, 0.f);
            term(xv[u].x, cv[u].x);
            term(xv[u].y, cv[u].y);
            term(xv[u].z, cv[u].z);
            term(xv[u].w, cv[u].w);
          }
          if (L == 32 && (terms += 4 * U) >= kSegTerms) widen();  // (fewer lanes: at most kSegTerms a segment)
        }
      } else {
        // a test per term keeps the loads apart (200,000 x 210: 116 -> 230 us), one per row still some
        // (122): one per U rows where their terms fit, else per piece of a row
        const int cnt = (n + L - 1) / L;
        const bool fit = L < 32 || U * cnt <= kSegTerms;
        if (L == 32 && fit) {
          if (terms + U * cnt > kSegTerms) widen();
          terms += U * cnt;
        }
#pragma unroll
        for (int u = 0; u < U; ++u) {
          if (id[u] < 0) continue;
          const float* x = data + (size_t)(s0 + (i + u) * G + grp) * n;
          const float* c = centers + (size_t)id[u] * n;
          if (fit) {
            for (int t = sub; t < n; t += L) term(ld(x + t), ld(c + t));
          } else {
            for (int b0 = 0; b0 < n; b0 += kSegTerms * L) {
              const int e = min(n, b0 + kSegTerms * L);
              if (terms > 0) widen();
              for (int t = b0 + sub; t < e; t += L) term(ld(x + t), ld(c + t));
              terms = kSegTerms;
            }
          }
        }
      }
#pragma unroll
      for (int u = 0; u < U; ++u) id[u] = nx[u];
    }
    if (L == 32) {
      if (terms > 0) widen();
      if (!off) {
        acc += seg;
        continue;
      }
    } else if (hi < 1e37f && (hi > 1e-24f || mx == 0.0f)) {
      acc += (double)hi + (double)lo;
      continue;
    }
    for (int i = 0; i < kSegSteps; ++i) {
      const long long r = s0 + i * G + grp;
      if (r >= m) continue;
      const float* x = data + (size_t)r * n;
      const float* c = centers + (size_t)ld(idx + r) * n;
      for (int t0 = vec ? 4 * sub : sub; t0 < n; t0 += vec ? 4 * L : L)
        for (int t = t0; t < t0 + (vec ? 4 : 1); ++t) {
          const double u = (double)x[t] - (double)c[t];
          acc = fma(u, u, acc);
        }
    }
  }
  const double t = block_sum(acc);
  if (threadIdx.x == 0) partial[blockIdx.x] = t;
}

// FP64 data: two FP64 operations per element (the lanes' sums meet once, at the end).
__global__ void __launch_bounds__(256)
compactness_d_kernel(long long m, int n, const double* data, const int* idx,
                     const double* centers, double* __restrict__ partial) {
  if (grid_enter()) return;
  const int lane = threadIdx.x & 31;
  const long long w0 = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const long long nw = ((long long)gridDim.x * blockDim.x) >> 5;
  double acc = 0.0;
  constexpr int U = 4;  // rows in flight
  for (long long r0 = w0 * U; r0 < m; r0 += nw * U) {
    const double* x[U];
    const double* c[U];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const long long r = r0 + u < m ? r0 + u : m - 1;
      x[u] = data + (size_t)r * n;
      c[u] = centers + (size_t)ld(idx + r) * n;
    }
    for (int t = lane; t < n; t += 32) {
      double v[U];
#pragma unroll
      for (int u = 0; u < U; ++u) v[u] = ld(x[u] + t) - ld(c[u] + t);
#pragma unroll
      for (int u = 0; u < U; ++u)
        if (r0 + u < m) acc = fma(v[u], v[u], acc);
    }
  }
  const double t = block_sum(acc);
  if (threadIdx.x == 0) partial[blockIdx.x] = t;
}

// One block: the partial sums, a strided chain per thread and a tree.
template <typename T>
__global__ void __launch_bounds__(256)
compactness_final_kernel(const double* partial, int nb, double* acc, T* out, bool last) {
  if (grid_enter()) return;
  double t = 0.0;
  for (int i = threadIdx.x; i < nb; i += 256) t += partial[i];
  t = block_sum(t);
  if (threadIdx.x == 0) {
    *acc += t;
    if (last) out[0] = (T)*acc;
  }
}

template <typename T>
__global__ void row_norm_kernel(int m0, int m, int n, const T* in, T* __restrict__ out) {
  if (grid_enter()) return;
  const int warps = blockDim.x >> 5, w = threadIdx.x >> 5, lane = threadIdx.x & 31;
  for (long long i = (long long)blockIdx.x * warps + w; i < m; i += (long long)gridDim.x * warps) {
    double s = 0.0;
    for (int t = lane; t < n; t += 32) s = fma((double)in[(size_t)i * n + t], (double)in[(size_t)i * n + t], s);
    for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    if (lane == 0) out[m0 + i] = (T)s;
  }
}

// 32 columns per block (coalesced rows), up to 32 threads a column, 16 rows or more each (strided); their
// FP64 chains are added in order. (One thread per column walked the rows alone: 128 x 256 took 23 us.
// Fewer rows a thread would round every square on its own: up to 16 rows stay one chain.)
template <typename T>
__global__ void __launch_bounds__(1024)
col_norm_kernel(int m, int n, const T* in, T* __restrict__ out) {
  if (grid_enter()) return;
  __shared__ double red[32][33];
  const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
  const long long j = (long long)blockIdx.x * 32 + tx;
  double s = 0.0;
  const int slices = min(32, (m + 15) / 16);
  if (j < n && ty < slices) {
#pragma unroll 8
    for (long long i = ty; i < m; i += slices) {
      const double v = (double)ld(in + (size_t)i * n + j);
      s = fma(v, v, s);
    }
  }
  red[ty][tx] = s;
  __syncthreads();
  if (ty == 0 && j < n) {
    double t = 0.0;
    for (int i = 0; i < slices; ++i) t += red[i][tx];
    out[j] = (T)t;
  }
}

// C = A B for row-major A (ra x ca), B (ca x cb) and C (ra x cb): 64 x 64 outputs per block of
// 256 threads (4 x 4 per thread), k in steps of 16 through shared memory; each output is one FMA
// chain over k in ascending order. Row tiles beyond the grid's y extent are taken in turn.
template <typename T>
__global__ void matmul_kernel(int ra, int ca, int cb, const T* A,
                              const T* B, T* __restrict__ C) {
  if (grid_enter()) return;
  constexpr int TM = 64, TN = 64, TK = 16;
  __shared__ T As[TK][TM + 1];
  __shared__ T Bs[TK][TN];
  const int tx = threadIdx.x % 16, ty = threadIdx.x / 16;
  const long long c0 = (long long)blockIdx.x * TN;
  const long long row_tiles = ((long long)ra + TM - 1) / TM;
  for (long long rt = blockIdx.y; rt < row_tiles; rt += gridDim.y) {
    const long long r0 = rt * TM;
    T acc[4][4];
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int j = 0; j < 4; ++j) acc[i][j] = T(0);
    for (int k0 = 0; k0 < ca; k0 += TK) {
      for (int e = threadIdx.x; e < TM * TK; e += blockDim.x) {
        const int rr = e / TK, kk = e % TK;
        const long long r = r0 + rr;
        As[kk][rr] = (r < ra && k0 + kk < ca) ? A[r * ca + k0 + kk] : T(0);
      }
      for (int e = threadIdx.x; e < TK * TN; e += blockDim.x) {
        const int kk = e / TN, cc = e % TN;
        const long long c = c0 + cc;
        Bs[kk][cc] = (k0 + kk < ca && c < cb) ? B[(long long)(k0 + kk) * cb + c] : T(0);
      }
      __syncthreads();
      const int kn = min(TK, ca - k0);
      for (int kk = 0; kk < kn; ++kk) {
        T a[4], b[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) a[i] = As[kk][ty + 16 * i];
#pragma unroll
        for (int j = 0; j < 4; ++j) b[j] = Bs[kk][tx + 16 * j];
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
          for (int j = 0; j < 4; ++j) acc[i][j] = fma(a[i], b[j], acc[i][j]);
      }
      __syncthreads();
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const long long r = r0 + ty + 16 * i;
      if (r >= ra) continue;
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const long long c = c0 + tx + 16 * j;
        if (c < cb) C[r * cb + c] = acc[i][j];
      }
    }
  }
}

template <typename T>
kmeansCudaErrorStatus mat_mat_mult(int ra, int ca, const T* A, int cb, const T* B, T* C) {
  if (ra < 0 || ca < 0 || cb < 0) return ERROR_MATMATMULT;
  if (ra == 0 || cb == 0) return NO_ERROR;
  if (!C || (ca > 0 && (!A || !B))) return ERROR_MATMATMULT;
  const long long col_tiles = ((long long)cb + 63) / 64, row_tiles = ((long long)ra + 63) / 64;
  const dim3 grid((unsigned)col_tiles, (unsigned)(row_tiles < 65535 ? row_tiles : 65535));
  launch(matmul_kernel<T>, grid, 256, 0, kDefault)(ra, ca, cb, A, B, C);
  kmgb::count_launches(1);
  return cudaGetLastError() ? ERROR_MATMATMULT : NO_ERROR;
}

// Sizing (base null) or carving of one temporary allocation.
struct Carver {
  char* base = nullptr;
  size_t off = 0;
  template <typename T>
  void take(T** p, size_t count) {
    *p = base ? reinterpret_cast<T*>(base + off) : nullptr;
    off += (sizeof(T) * (count ? count : 1) + 255) / 256 * 256;
  }
};

// ClosestCentersF/D. The rows' arg-min of nb_j - 2 A_i.B_j, equal to the FP64 evaluation.
//
// Split BF16 tensor cores where the dimension allows and the scan is long enough to pay for the
// rows' BF16 planes (read once, written once) and some ten launches: FP32 from rows x centers (in
// chunks of 128, the FP32 kernel's) x dimensions of 2^28 on, where the FP32 scan takes 12 us; FP64,
// whose scan runs at 0.6 TFMA/s, from 2^24 on. The rows go through in chunks whose planes stay in L2
// (and bound the workspace), whole waves of the pair kernel each. What the certificate leaves open
// is settled from recorded candidates (float-float; FP64 data: FP64), the rest by the tiled stages
// (FP64 data: a scan of the listed rows). The call returns before its kernels have run, so a scan whose
// bounded wait gave up is not reported but made up for: the last kernel then takes every row. FP32 scan:
// 898,790 x 128, K=256 took 1.52 ms, its re-rank 0.28 ms; FP64 scan: 100,000 x 64, K=256 took 2.80 ms.
template <typename T>
cudaError_t closest_centers(int m0, long long n, int d, const T* A, int k, const T* B, const T* nb,
                            int* out) {
  constexpr bool kF32 = sizeof(T) == 4;
  const long long ld = (d + 3) / 4 * 4, ldb = (d + 7) / 8 * 8;
  const bool direct = ld == d && !(reinterpret_cast<uintptr_t>(A) & 15);  // FP32 kernels' layout
  const long long kp = (k + 127) / 128 * 128;
  bool tc = bf16_tc_supported(d, 2) && n >= 256 && n * kp >= (1LL << (kF32 ? 28 : 24)) / d;
  const bool tiled = rerank_tiled_supported(d);
  const int threads = 256;
  const size_t smem = sizeof(double) * (size_t)d * (threads / 32);  // closest_fp64_kernel's
  auto scan_fp64 = [&]() -> cudaError_t {
    launch(closest_fp64_kernel, kmgb::num_sms() * 8, threads, smem, kDefault)(
        m0, (int)n, d, reinterpret_cast<const double*>(A), k, reinterpret_cast<const double*>(B),
        reinterpret_cast<const double*>(nb), out, nullptr, nullptr, nullptr);
    count_launches(1);
    return cudaGetLastError();
  };
  if (!kF32 && !tc) return scan_fp64();
  bool copy = !tc && !direct;  // the FP32 scan reads 16-byte aligned rows
  const long long wave = 256LL * (num_sms() / 2);
  const long long chunk = std::min(n, wave * std::max(1LL, (96LL << 20) / (wave * ldb * 4)));
  const long long cap = std::min(n, std::max(1024LL, n / 8));
  float *Ap, *Bt, *nbx, *xn, *cmax, *cinit, *thr, *thrC;
  int *list, *over, *sc, *cand, *cand_cnt;
  char *Xb, *Xl, *XbC, *XlC, *Cb, *Cl, *cbias;
  const long long kpad = (k + kCenterPad - 1) / kCenterPad * kCenterPad;
  auto carve = [&](Carver& c) {
    c.take(&sc, 8);  // [0] cmax, [1] flagged, [2] left by the candidates, [4] error
    c.take(&Ap, copy ? n * ld : 0);
    c.take(&Bt, k * ld);
    c.take(&nbx, k);
    c.take(&xn, n);
    c.take(&list, n);
    c.take(&over, tc ? n : 0);
    if (!tc) return;
    c.take(&cinit, kpad);
    c.take(&cbias, kpad * kBiasCols * 2);
    c.take(&Cb, k * ldb * 2);
    c.take(&Cl, k * ldb * 2);
    c.take(&Xb, chunk * ldb * 2);
    c.take(&Xl, chunk * ldb * 2);
    c.take(&thr, n);
    c.take(&XbC, cap * ldb * 2);
    c.take(&XlC, cap * ldb * 2);
    c.take(&thrC, cap);
    c.take(&cand, cap * kMaxCand);
    c.take(&cand_cnt, cap);
  };
  cinit = thr = thrC = nullptr;
  Xb = Xl = XbC = XlC = Cb = Cl = cbias = nullptr;
  cand = cand_cnt = nullptr;
  Carver size;
  carve(size);
  void* mem = nullptr;
  cudaError_t e = call_alloc(&mem, size.off, kDefault);
  if (e == cudaErrorMemoryAllocation && tc) {
    // no room for the planes and candidates: the scans without them (FP64: without any memory)
    cudaGetLastError();
    if (!kF32) return scan_fp64();
    tc = false;
    copy = !direct;
    size = Carver{};
    carve(size);
    e = call_alloc(&mem, size.off, kDefault);
  }
  if (e) return e;
  Carver cut;
  cut.base = static_cast<char*>(mem);
  carve(cut);
  cmax = reinterpret_cast<float*>(sc);
  e = cudaMemsetAsync(sc, 0, 8 * sizeof(int), kDefault);
  const T* Xa = A;
  if (!e && copy) {
    launch(copy_pad_kernel, num_sms() * 8, 256, 0, kDefault)(reinterpret_cast<const float*>(A), n, d, Ap,
                                                         ld);
    count_launches(1);
    e = cudaGetLastError();
    Xa = reinterpret_cast<const T*>(Ap);
  }
  const long long ldx = copy ? ld : d;
  if (!e)
    e = launch_prep_expansion<T>(B, d, k, nb, Bt, ld, nbx, tc ? Cb : nullptr, Cl, ldb,
                                 tc ? cinit : nullptr, tc ? cbias : nullptr, cmax, kDefault);
  AssignArgs a{};
  a.cn = nbx;
  a.xnorm = xn;
  a.cmax = cmax;
  a.labels = out + m0;
  a.rerank_list = list;
  a.rerank_count = sc + 1;
  a.err = sc + 4;
  a.n = n;
  a.k = k;
  a.d = d;
  a.certify = 1;
  test_wait_hook(&a.test_withhold, &a.test_wait_cycles);  // zero unless a test asks
  if (tc) {
    a.gamma = assign_bf16_gamma(d);
    a.cinit = cinit;
    a.cbias = cbias;
    a.thr_out = thr;
    if (!kF32) a.pert = 0x1p-22f;  // FP32 roundings of FP64 rows and centers (computeKmeansD's bound)
    for (long long r0 = 0; r0 < n && !e; r0 += chunk) {
      const long long nr = std::min(chunk, n - r0);
      e = launch_prep_rows(Xa + (size_t)r0 * ldx, ldx, nr, d, nullptr, xn + r0, Xb, Xl, ldb, nullptr,
                           kDefault);
      AssignArgs ac = a;
      ac.n = nr;
      ac.out0 = r0;
      if (!e) e = launch_assign_bf16(Xb, Xl, ldb, Cb, Cl, ldb, ac, kDefault);
    }
    // the flagged rows again, recording their candidates
    RowList rl{list, sc + 1, thr, thrC, over, sc + 2};
    if (!e)
      e = launch_prep_rows(Xa, ldx, cap, d, nullptr, nullptr, XbC, XlC, ldb, nullptr, kDefault, nullptr,
                           &rl);
    AssignArgs c2 = a;
    c2.n = cap;
    c2.n_dev = sc + 1;
    c2.labels = nullptr;
    c2.certify = 0;
    c2.thr_out = nullptr;
    c2.thr_in = thrC;
    c2.cand = cand;
    c2.cand_cnt = cand_cnt;
    if (!e) e = launch_assign_bf16(XbC, XlC, ldb, Cb, Cl, ldb, c2, kDefault);
    if (!e && a.test_withhold) {  // (as a wait of the pair kernel that gave up would leave things)
      e = cudaMemsetAsync(sc + 4, 1, sizeof(int), kDefault);
      if (!e) e = cudaMemsetAsync(out + m0, 0xff, sizeof(int) * (size_t)n, kDefault);
    }
  } else {
    a.gamma = assign_fp32_gamma(d);
    if (!e)
      e = launch_prep_rows(Xa, ldx, n, d, nullptr, xn, nullptr, nullptr, 0, nullptr, kDefault);
    if (!e) e = launch_assign_fp32(reinterpret_cast<const float*>(Xa), ld, Bt, ld, a, kDefault);
  }
  if (kF32) {
    RerankArgs r{};
    r.X = reinterpret_cast<const float*>(Xa);
    r.ldx = ldx;
    r.C = Bt;
    r.ldc = ld;
    r.nb = nbx;
    r.xnorm = xn;
    r.cmax = cmax;
    r.list = list;
    r.count = sc + 1;
    r.labels = out + m0;
    r.n = n;
    r.k = k;
    r.d = d;
    r.mode = 1;
    r.max_list = tc ? cap : n;
    r.redo = sc + 4;
    if (!e && tc) e = launch_resolve_expansion(r, cand, cand_cnt, over, sc + 2, kDefault);
    if (tc) {
      r.list = over;
      r.count = sc + 2;
      r.max_list = n;
    }
    if (!e && tiled) {
      e = launch_rerank_settle(r, kDefault);
    } else if (!e) {
      e = launch_rerank(r, kDefault);
    }
  } else {
    ResolveD r{};
    r.X = reinterpret_cast<const double*>(A);
    r.ldx = d;
    r.C = reinterpret_cast<const double*>(B);
    r.c_dim = k;
    r.c_row = 1;
    r.nb = reinterpret_cast<const double*>(nb);
    r.d = d;
    r.k = k;
    r.mode = 1;
    r.list = list;
    r.count = sc + 1;
    r.max_list = cap;
    r.cand = cand;
    r.cand_cnt = cand_cnt;
    r.labels = out + m0;
    r.over = over;
    r.over_count = sc + 2;
    if (!e) e = launch_resolve_fp64(r, kDefault);
    if (!e) {
      launch(closest_fp64_kernel, num_sms() * 8, threads, smem, kDefault)(
          m0, (int)n, d, r.X, k, r.C, r.nb, out, over, sc + 2, sc + 4);
      count_launches(1);
      e = cudaGetLastError();
    }
  }
  call_free(mem, kDefault);
  return e;
}

template <typename T>
kmeansCudaErrorStatus cluster_centers(int m0, int m, int n, int k, bool lastTile, const T* data,
                                      const int* indices, T* centers_large, int* counts_large,
                                      T* centers, int* counts) {
  if (m < 0 || n <= 0 || k <= 0 || !centers_large || !counts_large) return ERROR_CLUSTERCENTERS;
  double* acc = reinterpret_cast<double*>(centers_large);
  if (reinterpret_cast<uintptr_t>(acc) & 7) return ERROR_CLUSTERCENTERS;
  UpdateWork w{};
  w.n = m;
  w.k = k;
  w.d = n;
  w.ldx = n;
  plan_update_tiles_fine(m, k, &w.tile_pts, &w.ntiles);
  w.max_pieces = m / kSumPiece + k + 1;
  const long long hist_elems = (long long)k * w.ntiles;
  cudaError_t e = cudaSuccess;
  if (m > 0) {
    e = tmp_alloc(&w.hist, hist_elems);
    if (!e) e = tmp_alloc(&w.label_off, k + 1);
    if (!e) e = tmp_alloc(&w.piece_cnt, k + 1);
    if (!e) e = tmp_alloc(&w.sorted, m);
    if (!e) e = tmp_alloc(&w.tickets, 1);
    if (!e) e = cudaMemsetAsync(w.tickets, 0, sizeof(int), kDefault);
    if (!e) e = tmp_alloc(&w.part, (size_t)w.max_pieces * n);
    if (!e) e = launch_tile_accumulate<T>(data, n, indices + m0, w, acc, counts_large, kDefault);
  }
  if (!e && lastTile) e = launch_finalize_acc<T>(acc, counts_large, k, n, centers, counts, kDefault);
  tmp_free(w.hist);
  tmp_free(w.label_off);
  tmp_free(w.piece_cnt);
  tmp_free(w.sorted);
  tmp_free(w.tickets);
  tmp_free(w.part);
  return e ? ERROR_CLUSTERCENTERS : NO_ERROR;
}

void launch_compactness(long long m, int n, const float* data, const int* idx, const float* centers,
                        double* part, int blocks) {
  const bool vec = n % 4 == 0 && !(reinterpret_cast<uintptr_t>(data) & 15) &&
                   !(reinterpret_cast<uintptr_t>(centers) & 15);
  const int per = vec ? (n + 3) / 4 : n;  // lanes' worth of a row
  auto kern = per <= 4 ? compactness_ff_kernel<4>
                       : (per <= 8 ? compactness_ff_kernel<8>
                                   : (per <= 16 ? compactness_ff_kernel<16> : compactness_ff_kernel<32>));
  launch(kern, blocks, 256, 0, kDefault)(m, n, data, idx, centers, vec, part);
  count_launches(1);
}
void launch_compactness(long long m, int n, const double* data, const int* idx, const double* centers,
                        double* part, int blocks) {
  launch(compactness_d_kernel, blocks, 256, 0, kDefault)(m, n, data, idx, centers, part);
  count_launches(1);
}

template <typename T>
kmeansCudaErrorStatus compactness(int m0, int m, bool lastTile, int n, int k, const T* data,
                                  const int* indices, const T* centers, T* out) {
  (void)k;
  if (m < 0 || n <= 0 || !out) return ERROR_COMPACTNESS;
  double* acc = (sizeof(T) == 4) ? reinterpret_cast<double*>(out + 2) : reinterpret_cast<double*>(out + 1);
  if (reinterpret_cast<uintptr_t>(acc) & 7) return ERROR_COMPACTNESS;
  const int blocks = kmgb::num_sms() * 8;
  double* part = nullptr;
  cudaError_t e = tmp_alloc(&part, blocks);
  if (!e) {
    launch_compactness(m, n, data, indices + m0, centers, part, blocks);
    e = cudaGetLastError();
  }
  if (!e) {
    launch(compactness_final_kernel<T>, 1, 256, 0, kDefault)(part, blocks, acc, out, lastTile);
    kmgb::count_launches(1);
    e = cudaGetLastError();
  }
  tmp_free(part);
  return e ? ERROR_COMPACTNESS : NO_ERROR;
}

}  // namespace

extern "C" {

kmeansCudaErrorStatus ClosestCentersF(const int m0, const int nRowsA, const int nColsA,
                                      const float* A, const int nColsB, const float* B,
                                      float* Bpadded, const float* normRowsOfA_squared,
                                      const float* normColsOfB_squared, const int nColsC, float* C,
                                      int* Cindices, int* CindicesFinal) {
  (void)Bpadded;
  (void)normRowsOfA_squared;
  (void)nColsC;
  (void)C;
  (void)Cindices;
  if (nRowsA < 0 || nColsA <= 0 || nColsB <= 0 || !A || !B || !normColsOfB_squared ||
      !CindicesFinal)
    return ERROR_CLOSESTCENTERS;
  if (nRowsA == 0) return NO_ERROR;
  return closest_centers<float>(m0, nRowsA, nColsA, A, nColsB, B, normColsOfB_squared, CindicesFinal)
             ? ERROR_CLOSESTCENTERS
             : NO_ERROR;
}

kmeansCudaErrorStatus ClosestCentersD(const int m0, const int nRowsA, const int nColsA,
                                      const double* A, const int nColsB, const double* B,
                                      double* Bpadded, const double* normRowsOfA_squared,
                                      const double* normColsOfB_squared, const int nColsC,
                                      double* C, int* Cindices, int* CindicesFinal) {
  (void)Bpadded;
  (void)normRowsOfA_squared;
  (void)nColsC;
  (void)C;
  (void)Cindices;
  if (nRowsA < 0 || nColsA <= 0 || nColsB <= 0 || !A || !B || !normColsOfB_squared ||
      !CindicesFinal)
    return ERROR_CLOSESTCENTERS;
  if (nRowsA == 0) return NO_ERROR;
  const int threads = 256;
  const size_t smem = sizeof(double) * nColsA * (threads / 32);
  if (smem > 200 * 1024) return ERROR_CLOSESTCENTERS;
  if (smem > 48 * 1024 &&
      cudaFuncSetAttribute(closest_fp64_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                           200 * 1024) != cudaSuccess)
    return ERROR_CLOSESTCENTERS;
  return closest_centers<double>(m0, nRowsA, nColsA, A, nColsB, B, normColsOfB_squared,
                                 CindicesFinal)
             ? ERROR_CLOSESTCENTERS
             : NO_ERROR;
}

kmeansCudaErrorStatus rowTransformMinimumF(const int m0, const int m, const int n,
                                           const float* normRowsOfA_squared,
                                           const float* normColsOfB_squared, const float* input,
                                           int* output) {
  if (m < 0 || n <= 0) return ERROR_ROWTRANSFORMMINIMUM;
  if (m == 0) return NO_ERROR;
  launch(row_transform_min_kernel<float>, kmgb::num_sms() * 8, 256, 0, kDefault)(
      m0, m, n, normRowsOfA_squared, normColsOfB_squared, input, output); kmgb::count_launches(1);
  return cudaGetLastError() ? ERROR_ROWTRANSFORMMINIMUM : NO_ERROR;
}

kmeansCudaErrorStatus rowTransformMinimumD(const int m0, const int m, const int n,
                                           const double* normRowsOfA_squared,
                                           const double* normColsOfB_squared,
                                           const double* input, int* output) {
  if (m < 0 || n <= 0) return ERROR_ROWTRANSFORMMINIMUM;
  if (m == 0) return NO_ERROR;
  launch(row_transform_min_kernel<double>, kmgb::num_sms() * 8, 256, 0, kDefault)(
      m0, m, n, normRowsOfA_squared, normColsOfB_squared, input, output); kmgb::count_launches(1);
  return cudaGetLastError() ? ERROR_ROWTRANSFORMMINIMUM : NO_ERROR;
}

kmeansCudaErrorStatus ClusterCentersF(const int m0, const int m, const int n, const int k,
                                      const bool lastTile, const float* data, const int* indices,
                                      float* centers_large, int* counts_large, float* centers,
                                      int* counts) {
  return cluster_centers<float>(m0, m, n, k, lastTile, data, indices, centers_large, counts_large,
                                centers, counts);
}

kmeansCudaErrorStatus ClusterCentersD(const int m0, const int m, const int n, const int k,
                                      const bool lastTile, const double* data, const int* indices,
                                      double* centers_large, int* counts_large, double* centers,
                                      int* counts) {
  return cluster_centers<double>(m0, m, n, k, lastTile, data, indices, centers_large,
                                 counts_large, centers, counts);
}

kmeansCudaErrorStatus CompactnessF(const int m0, const int m, const bool lastTile, const int n,
                                   const int k, const float* data, const int* indices,
                                   const float* centers, float* compactness_out) {
  return compactness<float>(m0, m, lastTile, n, k, data, indices, centers, compactness_out);
}

kmeansCudaErrorStatus CompactnessD(const int m0, const int m, const bool lastTile, const int n,
                                   const int k, const double* data, const int* indices,
                                   const double* centers, double* compactness_out) {
  return compactness<double>(m0, m, lastTile, n, k, data, indices, centers, compactness_out);
}

kmeansCudaErrorStatus MatMatMultF(const int nRowsA, const int nColsA, const float* A,
                                  const int nColsB, const float* B, float* C) {
  return mat_mat_mult<float>(nRowsA, nColsA, A, nColsB, B, C);
}

kmeansCudaErrorStatus MatMatMultD(const int nRowsA, const int nColsA, const double* A,
                                  const int nColsB, const double* B, double* C) {
  return mat_mat_mult<double>(nRowsA, nColsA, A, nColsB, B, C);
}

kmeansCudaErrorStatus rowNormalizeF(const int m0, const int m, const int n, const float* input,
                                    float* output) {
  if (m < 0 || n <= 0) return ERROR_ROWNORMALIZE;
  if (m == 0) return NO_ERROR;
  return launch_row_norms(input, n, m, n, output + m0, kDefault) ? ERROR_ROWNORMALIZE : NO_ERROR;
}

kmeansCudaErrorStatus rowNormalizeD(const int m0, const int m, const int n, const double* input,
                                    double* output) {
  if (m < 0 || n <= 0) return ERROR_ROWNORMALIZE;
  if (m == 0) return NO_ERROR;
  launch(row_norm_kernel<double>, kmgb::num_sms() * 8, 256, 0, kDefault)(m0, m, n, input, output);
  kmgb::count_launches(1);
  return cudaGetLastError() ? ERROR_ROWNORMALIZE : NO_ERROR;
}

kmeansCudaErrorStatus colNormalizeF(const int m, const int n, const float* input, float* output) {
  if (m < 0 || n <= 0) return ERROR_COLNORMALIZE;
  launch(col_norm_kernel<float>, (unsigned)(((long long)n + 31) / 32), 1024, 0, kDefault)(m, n, input,
                                                                                         output);
  kmgb::count_launches(1);
  return cudaGetLastError() ? ERROR_COLNORMALIZE : NO_ERROR;
}

kmeansCudaErrorStatus colNormalizeD(const int m, const int n, const double* input,
                                    double* output) {
  if (m < 0 || n <= 0) return ERROR_COLNORMALIZE;
  launch(col_norm_kernel<double>, (unsigned)(((long long)n + 31) / 32), 1024, 0, kDefault)(m, n, input,
                                                                                          output);
  kmgb::count_launches(1);
  return cudaGetLastError() ? ERROR_COLNORMALIZE : NO_ERROR;
}

}  // extern "C"
