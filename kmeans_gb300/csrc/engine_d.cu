// computeKmeansD: the reference's double-precision driver entry (main/cpp/kmeans.cpp:1364-1409).
//
// The reference's FP64 custom assignment is broken (its partial reduction for double2 is an
// empty function, main/cuda/reduction.hcu:7-11, so every label becomes 0); only its cuBLAS path
// (cublasDgemm + rowTransformMinimumD, kmeans.cpp:958-993) defines FP64 behaviour. This path
// computes what that one intends, exactly: label = FP64 arg-min of sum_d (x_d - c_d)^2 (lowest
// index on ties), centers = canonical FP64 sums / counts, SSE in FP64 against the new centers.
// FP64 throughput on GB300 is low (about 1.25 TFLOP/s): full batches take the tensor cores as a
// filter on FP32 roundings and settle the few open rows from recorded candidates in FP64, and the
// update and the SSE, two FP64 operations per element, run over the clusters whose members changed.
#include <algorithm>
#include <cmath>
#include <cstdint>
#include <cstdlib>
#include <cstring>
#include <future>
#include <random>
#include <string>
#include <vector>

#include "../../include/kmeans_gb300.h"
#include "common.cuh"
#include "kernels.h"

using namespace kmgb;

namespace {

// CT[t][j] = C[j][t]
__global__ void transpose_d_kernel(const double* C, int k, int d, double* __restrict__ CT) {
  if (grid_enter()) return;
  const long long total = (long long)k * d;
  for (long long e = (long long)blockIdx.x * blockDim.x + threadIdx.x; e < total;
       e += (long long)gridDim.x * blockDim.x) {
    const int j = (int)(e / d), t = (int)(e % d);
    CT[(size_t)t * k + j] = C[e];
  }
}

// One warp per point, lanes over centers (coalesced reads of CT); exact FP64 direct distance.
// list (nullable): only the points list[0 .. *count) (the tensor pass's uncertified points).
__global__ void assign_d_kernel(const double* X, long long n, int d,
                                const double* CT, int k, int* __restrict__ labels,
                                const int* list,
                                const int* count) {
  if (grid_enter()) return;
  extern __shared__ double xs_all[];
  const int warps = blockDim.x >> 5, w = threadIdx.x >> 5, lane = threadIdx.x & 31;
  double* xs = xs_all + (size_t)w * d;
  const long long todo = list ? (long long)*count : n;
  for (long long slot = (long long)blockIdx.x * warps + w; slot < todo;
       slot += (long long)gridDim.x * warps) {
    const long long i = list ? (long long)list[slot] : slot;
    for (int t = lane; t < d; t += 32) xs[t] = X[(size_t)i * d + t];
    __syncwarp();
    double best = INFINITY;
    int bi = -1;
    for (int j = lane; j < k; j += 32) {
      double s = 0.0;
      for (int t = 0; t < d; ++t) {
        const double u = xs[t] - CT[(size_t)t * k + j];
        s = fma(u, u, s);
      }
      if (s < best) {
        best = s;
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
    if (lane == 0) labels[i] = bi < 0 ? 0 : bi;
    __syncwarp();
  }
}

// out[r][c] = (float)in[r][c] (round to nearest) for c < d, 0 for d <= c < ldo.
__global__ void d2f_kernel(const double* in, long long rows, int d,
                           float* __restrict__ out, long long ldo) {
  if (grid_enter()) return;
  const long long total = rows * ldo;
  for (long long e = (long long)blockIdx.x * blockDim.x + threadIdx.x; e < total;
       e += (long long)gridDim.x * blockDim.x) {
    const long long r = e / ldo, c = e - r * ldo;
    out[e] = c < d ? __double2float_rn(in[(size_t)r * d + c]) : 0.0f;
  }
}

// SSE against the new centers, by the pieces of the label-sorted rows (kSumPiece rows of one cluster
// each, as the canonical sums): one warp per piece, lanes over the dimensions, four rows in flight;
// the lanes meet once per piece.
__global__ void __launch_bounds__(128)
sse_pieces_kernel(const double* X, int d, const int* sorted,
                  const int* label_off, const int* pstart, int k,
                  const double* C, double* __restrict__ piece) {
  if (grid_enter()) return;
  const int total = pstart[k];
  const int lane = threadIdx.x & 31;
  const int nw = (int)((gridDim.x * blockDim.x) >> 5);
  constexpr int U = 4;
  for (int p = (int)((blockIdx.x * blockDim.x + threadIdx.x) >> 5); p < total; p += nw) {
    int lo = 0, hi = k - 1;  // the cluster of piece p
    while (lo < hi) {
      const int mid = (lo + hi + 1) >> 1;
      if (ld(pstart + mid) <= p) lo = mid;
      else hi = mid - 1;
    }
    const int b = label_off[lo] + (p - pstart[lo]) * kSumPiece;
    const int e = min(b + kSumPiece, label_off[lo + 1]);
    const double* c = C + (size_t)lo * d;
    double acc = 0.0;
    for (int t0 = b; t0 < e; t0 += 32) {
      const int ids = t0 + lane < e ? ld(sorted + t0 + lane) : 0;
      const int cnt = min(32, e - t0);
      for (int h = 0; h < cnt; h += U) {
        const double* x[U];
#pragma unroll
        for (int u = 0; u < U; ++u)
          x[u] = X + (size_t)__shfl_sync(0xffffffffu, ids, min(h + u, cnt - 1)) * d;
        for (int t = lane; t < d; t += 32) {
          const double cv = ld(c + t);
          double v[U];
#pragma unroll
          for (int u = 0; u < U; ++u) v[u] = ld(x[u] + t) - cv;
#pragma unroll
          for (int u = 0; u < U; ++u)
            if (h + u < cnt) acc = fma(v[u], v[u], acc);
        }
      }
    }
    for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
    if (lane == 0) piece[p] = acc;
  }
}

// One block: every cluster's SSE from its pieces (in order; a cluster without pieces in this
// iteration keeps its value), and their sum.
__global__ void __launch_bounds__(1024)
sse_d_final_kernel(const double* piece, const int* pstart, int k,
                   const int* dirty, double* __restrict__ sse_k, double* out) {
  if (grid_enter()) return;
  __shared__ double red[1024];
  double t = 0.0;
  for (int j = threadIdx.x; j < k; j += 1024) {
    if (!dirty || dirty[j]) {
      double s = 0.0;
      const int p1 = pstart[j + 1];
#pragma unroll 4
      for (int p = pstart[j]; p < p1; ++p) s += piece[p];
      sse_k[j] = s;
    }
    t += sse_k[j];
  }
  red[threadIdx.x] = t;
  __syncthreads();
  for (int w = 512; w > 0; w >>= 1) {
    if ((int)threadIdx.x < w) red[threadIdx.x] += red[threadIdx.x + w];
    __syncthreads();
  }
  if (threadIdx.x == 0) *out = red[0];
}

__global__ void gather_d_kernel(const double* X, int d, const int* perm,
                                long long m, long long start, long long m_mb, double* __restrict__ Xw) {
  if (grid_enter()) return;
  const long long total = m_mb * d;
  for (long long e = (long long)blockIdx.x * blockDim.x + threadIdx.x; e < total;
       e += (long long)gridDim.x * blockDim.x) {
    const long long r = e / d;
    long long pos = start + r;
    if (pos >= m) pos -= m;
    Xw[e] = X[(size_t)perm[pos] * d + (e % d)];
  }
}

// Device buffers from the library's pool (a call's some twenty cudaMalloc and cudaFree, each of
// which waits for the device, took about 2 ms), given back when the call ends.
struct DevBufs {
  std::vector<void*> ptrs;
  ~DevBufs() {
    cudaStreamSynchronize(0);
    for (void* p : ptrs) call_free(p, 0);
  }
  template <typename T>
  cudaError_t alloc(T** p, size_t count) {
    void* v = nullptr;
    const cudaError_t e = call_alloc(&v, sizeof(T) * (count ? count : 1), 0);
    *p = static_cast<T*>(v);
    if (e == cudaSuccess) ptrs.push_back(v);
    return e;
  }
  // Buffers a call can do without: all that `take` allocates, or none of it.
  template <typename F>
  bool optional(F take) {
    const size_t had = ptrs.size();
    if (take()) return true;
    cudaGetLastError();
    for (; ptrs.size() > had; ptrs.pop_back()) call_free(ptrs.back(), 0);
    return false;
  }
};

#define KD_TRY(expr, code)                \
  do {                                    \
    if ((expr) != cudaSuccess) return (code); \
  } while (0)

// Distance bounds: as the FP32-data engine's, but from a fifth of its work on, since here the FP64
// sums and SSE of the unchanged clusters are saved as well (400,000 x 64, K=256).
bool prune_worthwhile(long long m, int k, int d) {
  const long long kp = (k + kCenterPad - 1) / kCenterPad * kCenterPad;
  return prune_enabled() && k >= 2 && (long long)k * 32 <= m && m * kp >= (1LL << 31) / d;
}

// The bounds' buffers; where they do not fit, every iteration scans every row.
void alloc_prune_d(DevBufs& B, PruneState* out, int** crr, long long m, int k, long long ldb) {
  PruneState p;
  p.n = m;
  p.k = k;
  p.cap = (int)std::min(m * 13 / 20, (8LL << 30) / (ldb * 4));
  if (p.cap < 256) return;
  uint16_t *xc = nullptr, *xlc = nullptr;
  auto got = [&](auto** q, size_t count) { return B.alloc(q, count) == cudaSuccess; };
  if (!B.optional([&] {
        return got(&p.ub, m) && got(&p.lb, m) && got(&p.shift, k) && got(&p.cxn, k) && got(&p.cub, k) &&
               got(&p.clb, k) && got(&p.clab, k) && got(crr, k) && got(&p.list, p.cap) &&
               got(&p.lab_old, m) && got(&p.dirty, k) && got(&p.flags, 8) && got(&p.top, 2) &&
               got(&xc, (size_t)p.cap * ldb) && got(&xlc, (size_t)p.cap * ldb) &&
               cudaMemsetAsync(p.flags, 0, 8 * sizeof(int), 0) == cudaSuccess;
      }))
    return;
  p.Xc = xc;
  p.Xlc = xlc;
  *out = p;
}

// One FP64 run. kpp_seed < 0: the reference initialisation; else k-means++ with that seed (on the
// device, from the uploaded data). result receives the initial then the final centers (D x K);
// *final_sse the SSE of the last iteration (NaN when none ran).
kmeansErrorStatus run_d(const double* data, int m, int n, int k, double criterion, int maxIters,
                        double* result, double fraction, long long kpp_seed, double* final_sse) {
  *final_sse = std::nan("");
  const bool mini = fraction < 1.0;
  const long long m_mb = mini ? (long long)(int)((float)fraction * (float)m) : m;
  if (m_mb <= 0) return KMEANS_ERROR_TILING;
  // reference initialisation on the host (kmeans.cpp:554-564, 876-888): the shuffle is
  // sequential and independent of the data, so it runs on a host thread while the data set is
  // allocated and uploaded
  struct RefInit {
    std::vector<int> perm, picks;
    bool ok = true;
  };
  auto ref_task = [m, k, kpp_seed] {
    RefInit r;
    reference_perm(m, r.perm);
    if (kpp_seed < 0) r.ok = reference_picks(m, k, r.picks);
    return r;
  };
  std::future<RefInit> ref;
  try {
    ref = std::async(std::launch::async, ref_task);
  } catch (...) {  // no thread to be had: run it when the result is asked for
    ref = std::async(std::launch::deferred, ref_task);
  }

  DevBufs B;
  double *X = nullptr, *Xw = nullptr, *Cd = nullptr, *CT = nullptr, *acc = nullptr, *part = nullptr,
         *sse = nullptr, *sse_k = nullptr;
  int *lab = nullptr, *cnt = nullptr, *permd = nullptr;
  const cudaStream_t s = 0;
  const kmeansErrorStatus E = KMEANS_ERROR_BUILDDATA;
  KD_TRY(B.alloc(&X, (size_t)m * n), E);
  KD_TRY(cudaMemcpy(X, data, sizeof(double) * (size_t)m * n, cudaMemcpyHostToDevice), E);

  RefInit r;
  try {
    r = ref.get();
  } catch (...) {
    return KMEANS_ERROR_INITIALIZE;
  }
  if (!r.ok) return KMEANS_ERROR_INITIALIZE;
  const std::vector<int>& perm = r.perm;
  const std::vector<int>& picks = r.picks;
  std::vector<double> C((size_t)k * n);
  if (kpp_seed < 0)
    for (int i = 0; i < k; ++i)
      for (int j = 0; j < n; ++j) {
        C[(size_t)i * n + j] = data[(size_t)perm[picks[i]] * n + j];
        result[(size_t)j * k + i] = C[(size_t)i * n + j];
      }
  if (mini) {
    KD_TRY(B.alloc(&Xw, (size_t)m_mb * n), E);
    KD_TRY(B.alloc(&permd, m), E);
    KD_TRY(cudaMemcpy(permd, perm.data(), sizeof(int) * m, cudaMemcpyHostToDevice), E);
  }
  KD_TRY(B.alloc(&Cd, (size_t)k * n), E);
  KD_TRY(B.alloc(&CT, (size_t)k * n), E);
  KD_TRY(B.alloc(&acc, (size_t)k * n), E);
  KD_TRY(B.alloc(&cnt, k), E);
  KD_TRY(B.alloc(&lab, m_mb), E);
  KD_TRY(B.alloc(&sse, 1), E);
  if (kpp_seed < 0) {
    KD_TRY(cudaMemcpy(Cd, C.data(), sizeof(double) * C.size(), cudaMemcpyHostToDevice), E);
  } else {
    KppWork<double> kw;
    int *kp = nullptr, *err = nullptr;
    const kmeansErrorStatus EI = KMEANS_ERROR_INITIALIZE;
    KD_TRY(B.alloc(&kw.d2, kmeanspp_d2_elems(m)), EI);
    KD_TRY(B.alloc(&kw.blocksum, kmeanspp_blocks(m)), EI);
    KD_TRY(B.alloc(&kw.scalars, kKppScalars), EI);
    if (!B.optional([&] {
          return B.alloc(&kw.near, m) == cudaSuccess && B.alloc(&kw.cc, k) == cudaSuccess;
        }))
      kw.near = nullptr, kw.cc = nullptr;  // every draw reads every row
    KD_TRY(B.alloc(&kp, k), EI);
    KD_TRY(B.alloc(&err, 1), EI);
    KD_TRY(cudaMemset(err, 0, sizeof(int)), EI);
    KD_TRY(launch_kmeanspp(X, n, m, n, k, (unsigned long long)kpp_seed, Cd, n, kp, kw, err, s),
           EI);
    KD_TRY(cudaMemcpy(C.data(), Cd, sizeof(double) * C.size(), cudaMemcpyDeviceToHost), EI);
    int e = 0;
    KD_TRY(cudaMemcpy(&e, err, sizeof(int), cudaMemcpyDeviceToHost), EI);
    if (e) return EI;
    for (int i = 0; i < k; ++i)
      for (int j = 0; j < n; ++j) result[(size_t)j * k + i] = C[(size_t)i * n + j];
  }
  UpdateWork w{};
  w.n = m_mb;
  w.k = k;
  w.d = n;
  w.ldx = n;
  plan_update_tiles_fine(m_mb, k, &w.tile_pts, &w.ntiles);
  w.max_pieces = m_mb / kSumPiece + k + 1;
  const long long hist_elems = (long long)k * w.ntiles;
  KD_TRY(B.alloc(&w.hist, hist_elems), E);
  KD_TRY(B.alloc(&w.label_off, k + 1), E);
  KD_TRY(B.alloc(&w.piece_cnt, k + 1), E);
  KD_TRY(B.alloc(&w.sorted, m_mb), E);
  KD_TRY(B.alloc(&w.part, (size_t)w.max_pieces * n), E);
  KD_TRY(B.alloc(&part, w.max_pieces), E);
  KD_TRY(B.alloc(&sse_k, k), E);
  KD_TRY(B.alloc(&w.tickets, 1), E);
  KD_TRY(cudaMemsetAsync(w.tickets, 0, sizeof(int), s), E);

  // Tensor path (full batches, D within the split tier's limit): X and the centers are rounded
  // to FP32, the split BF16 tier assigns every point under its bound widened by that rounding
  // (|key(x,c) - key(fl(x),fl(c))| <= 2^-23 (|x||c| + |c|^2/2), taken twice), and the points it
  // cannot certify get the exact FP64 scan. KMGB_ASSIGN=fp32 keeps the FP64 scan for every point.
  const char* tier_env = std::getenv("KMGB_ASSIGN");
  const bool tc = !mini && bf16_tc_supported(n, 2) &&
                  !(tier_env && std::strcmp(tier_env, "fp32") == 0);
  const long long ldx = (n + 3) / 4 * 4, ldb = (n + 7) / 8 * 8;
  float *xn = nullptr, *Cf = nullptr, *Cop = nullptr, *cn = nullptr,
        *cmax = nullptr, *cinit = nullptr;
  uint16_t *Xb = nullptr, *Xl = nullptr, *Cb = nullptr, *Cl = nullptr, *cbias = nullptr,
           *XbC = nullptr, *XlC = nullptr;
  float *thr = nullptr, *thrC = nullptr;
  int *rr_list = nullptr, *rr_count = nullptr, *derr = nullptr, *over = nullptr, *cand = nullptr,
      *cand_cnt = nullptr;
  // rows of the candidate pass's compact copies; flagged rows past it take the FP64 scan
  long long cap = std::min<long long>(m, std::max<long long>(1024, m / 8));
  PruneState pr;
  int* crr_list = nullptr;
  if (tc) {
    const kmeansErrorStatus EA = KMEANS_ERROR_CLOSEST_CENTERS;
    KD_TRY(B.alloc(&xn, m), E);
    KD_TRY(B.alloc(&Xb, (size_t)m * ldb), E);
    KD_TRY(B.alloc(&Xl, (size_t)m * ldb), E);
    KD_TRY(B.alloc(&Cf, (size_t)k * ldx), E);
    KD_TRY(B.alloc(&Cop, (size_t)k * ldx), E);
    KD_TRY(B.alloc(&Cb, (size_t)k * ldb), E);
    KD_TRY(B.alloc(&Cl, (size_t)k * ldb), E);
    KD_TRY(B.alloc(&cn, k), E);
    KD_TRY(B.alloc(&cmax, 1), E);
    KD_TRY(B.alloc(&cinit, (size_t)((k + kCenterPad - 1) / kCenterPad * kCenterPad)), E);
    KD_TRY(B.alloc(&cbias, (size_t)((k + kCenterPad - 1) / kCenterPad * kCenterPad) * kBiasCols), E);
    KD_TRY(B.alloc(&thr, m), E);
    KD_TRY(B.alloc(&over, m), E);
    KD_TRY(B.alloc(&rr_list, m), E);
    KD_TRY(B.alloc(&rr_count, 3), E);
    KD_TRY(B.alloc(&derr, 1), E);
    KD_TRY(cudaMemsetAsync(derr, 0, sizeof(int), s), E);
    // what can be smaller or missing comes last
    while (!B.optional([&] {
      return B.alloc(&thrC, cap) == cudaSuccess && B.alloc(&XbC, (size_t)cap * ldb) == cudaSuccess &&
             B.alloc(&XlC, (size_t)cap * ldb) == cudaSuccess &&
             B.alloc(&cand, (size_t)cap * kMaxCand) == cudaSuccess &&
             B.alloc(&cand_cnt, cap) == cudaSuccess;
    })) {
      if (cap <= 1024) return E;
      cap = std::max<long long>(1024, cap / 4);
    }
    if (maxIters > 1 && prune_worthwhile(m, k, n)) alloc_prune_d(B, &pr, &crr_list, m, k, ldb);
    KD_TRY(launch_prep_rows(X, n, m, n, nullptr, xn, Xb, Xl, ldb, nullptr, s), EA);
  }

  const int threads = 256;
  const size_t smem = sizeof(double) * n * (threads / 32);
  if (smem > 200 * 1024) return KMEANS_ERROR_CLOSEST_CENTERS;
  if (smem > 48 * 1024)
    KD_TRY(cudaFuncSetAttribute(assign_d_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                200 * 1024),
           KMEANS_ERROR_CLOSEST_CENTERS);
  double sse_old = 0.0, rel = 1.0;
  int it = 0;
  long long start = 0;
  while (it < maxIters && rel > criterion) {
    const double* Xa = X;
    if (mini) {
      launch(gather_d_kernel, kmgb::num_sms() * 8, 256, 0, s)(X, n, permd, m, start, m_mb, Xw);
      kmgb::count_launches(1);
      Xa = Xw;
    }
    launch(transpose_d_kernel, kmgb::num_sms() * 4, 256, 0, s)(Cd, k, n, CT); kmgb::count_launches(1);
    if (tc) {
      const kmeansErrorStatus EA = KMEANS_ERROR_CLOSEST_CENTERS;
      launch(d2f_kernel, kmgb::num_sms() * 4, 256, 0, s)(Cd, k, n, Cf, ldx); kmgb::count_launches(1);
      KD_TRY(cudaMemsetAsync(cmax, 0, sizeof(float), s), EA);
      KD_TRY(cudaMemsetAsync(rr_count, 0, 3 * sizeof(int), s), EA);
      KD_TRY(launch_prep_centers(Cf, ldx, k, n, Cop, Cb, ldb, cn, cmax, s, nullptr, cinit, Cl, cbias,
                                 pr.shift, pr.cxn, 0x1p-22f),
             EA);
      AssignArgs a{};
      a.cn = cn;
      a.xnorm = xn;
      a.cmax = cmax;
      a.cinit = cinit;
      a.cbias = cbias;
      a.thr_out = thr;
      a.labels = lab;
      a.rerank_list = rr_list;
      a.rerank_count = rr_count;
      a.err = derr;
      a.n = m;
      a.k = k;
      a.d = n;
      a.certify = 1;
      a.gamma = assign_bf16_gamma(n);
      a.pert = 0x1p-22f;
      AssignArgs af = a;
      if (pr.n > 0) {  // distance bounds (prune.cu)
        KD_TRY(launch_prune_top(pr, nullptr, s), EA);
        AssignArgs c = a;
        c.n = k;
        c.n_dev = pr.flags + 6;
        c.xnorm = pr.cxn;
        c.labels = pr.clab;
        c.rerank_list = crr_list;
        c.rerank_count = pr.flags + 2;
        c.thr_out = nullptr;
        c.ub = pr.cub;
        c.lb = pr.clb;
        KD_TRY(launch_assign_bf16(Cb, Cl, ldb, Cb, Cl, ldb, c, s), EA);
        KD_TRY(launch_prune_filter(pr, lab, nullptr, s), EA);
        KD_TRY(launch_prune_gather(pr, Xb, Xl, ldb * 2, nullptr, s), EA);
        af.ub = pr.ub;
        af.lb = pr.lb;
        af.sel = pr.flags + 1;
        af.sel_cap = pr.cap;
        af.row_map = pr.list;
        af.Xc = pr.Xc;
        af.Xlc = pr.Xlc;
      }
      KD_TRY(launch_assign_bf16(Xb, Xl, ldb, Cb, Cl, ldb, af, s), EA);
      // flagged rows: their candidates from a second pass, settled in FP64; rows without a record
      // take the FP64 scan (every flagged row scanned: 183 us an iteration at 400,000 x 64, K=256)
      KD_TRY(launch_gather_flagged(rr_list, rr_count, cap, Xb, Xl, ldb * 2, thr, XbC, XlC, thrC, over,
                                   rr_count + 1, nullptr, s),
             EA);
      AssignArgs c2 = a;
      c2.n = cap;
      c2.n_dev = rr_count;
      c2.labels = nullptr;
      c2.certify = 0;
      c2.thr_out = nullptr;
      c2.thr_in = thrC;
      c2.cand = cand;
      c2.cand_cnt = cand_cnt;
      KD_TRY(launch_assign_bf16(XbC, XlC, ldb, Cb, Cl, ldb, c2, s), EA);
      ResolveD rd{};
      rd.X = X;
      rd.ldx = n;
      rd.C = Cd;
      rd.c_dim = 1;
      rd.c_row = n;
      rd.d = n;
      rd.k = k;
      rd.mode = 0;
      rd.list = rr_list;
      rd.count = rr_count;
      rd.max_list = cap;
      rd.cand = cand;
      rd.cand_cnt = cand_cnt;
      rd.labels = lab;
      rd.over = over;
      rd.over_count = rr_count + 1;
      KD_TRY(launch_resolve_fp64(rd, s), EA);
      launch(assign_d_kernel, kmgb::num_sms() * 8, threads, smem, s)(X, m, n, CT, k, lab, over,
                                                                 rr_count + 1);
      kmgb::count_launches(1);
      if (pr.n > 0) {
        KD_TRY(launch_prune_dirty(pr, lab, nullptr, s), EA);
        w.dirty = pr.dirty;
      }
    } else {
      launch(assign_d_kernel, kmgb::num_sms() * 8, threads, smem, s)(Xa, m_mb, n, CT, k, lab, nullptr, nullptr);
      kmgb::count_launches(1);
    }
    KD_TRY(cudaGetLastError(), KMEANS_ERROR_CLOSEST_CENTERS);
    KD_TRY(cudaMemsetAsync(acc, 0, sizeof(double) * (size_t)k * n, s), KMEANS_ERROR_RESET);
    KD_TRY(cudaMemsetAsync(cnt, 0, sizeof(int) * k, s), KMEANS_ERROR_RESET);
    KD_TRY(launch_tile_accumulate<double>(Xa, n, lab, w, acc, cnt, s), KMEANS_ERROR_CLUSTER_CENTERS);
    KD_TRY(launch_finalize_acc<double>(acc, cnt, k, n, Cd, nullptr, s, w.dirty),
           KMEANS_ERROR_CLUSTER_CENTERS);
    launch(sse_pieces_kernel, kmgb::num_sms() * 8, 128, 0, s)(Xa, n, w.sorted, w.label_off, w.piece_cnt, k,
                                                          Cd, part);
    launch(sse_d_final_kernel, 1, 1024, 0, s)(part, w.piece_cnt, k, w.dirty, sse_k, sse);
    kmgb::count_launches(2);
    KD_TRY(cudaGetLastError(), KMEANS_ERROR_COMPACTNESS);
    double h = 0.0;
    KD_TRY(cudaMemcpy(&h, sse, sizeof(double), cudaMemcpyDeviceToHost), KMEANS_ERROR_COMPACTNESS);
    rel = std::fabs(h - sse_old) / std::fabs(h);
    sse_old = h;
    *final_sse = h;
    ++it;
    if (mini) {
      start += m_mb;
      if (start > m) start %= m;
      else if (start == m) start = 0;
    }
  }
  KD_TRY(cudaMemcpy(C.data(), Cd, sizeof(double) * C.size(), cudaMemcpyDeviceToHost),
         KMEANS_ERROR_GET_CENTERS);
  if (tc) {  // a bounded wait of the tensor pass gave up: its labels cannot be trusted
    int e = 0;
    KD_TRY(cudaMemcpy(&e, derr, sizeof(int), cudaMemcpyDeviceToHost), KMEANS_ERROR_CLOSEST_CENTERS);
    if (e) {
      set_last_error("computeKmeansD: a bounded wait in the tensor-core assignment gave up");
      return KMEANS_ERROR_CLOSEST_CENTERS;
    }
  }
  for (int i = 0; i < k; ++i)
    for (int j = 0; j < n; ++j) result[(size_t)j * k + i] = C[(size_t)i * n + j];
  return (rel <= criterion) ? KMEANS_SUCCESS : KMEANS_NONCONVERGENCE;
}

}  // namespace

extern "C" kmeansErrorStatus computeKmeansD(const double* data, const int m, const int n,
                                            const int k, const double criterion,
                                            const int maxIters, const int numRetries,
                                            const int initAlgorithm, const int doFullSGEMM,
                                            const int matrixFormat, double* result,
                                            const double miniBatchFraction) {
  if (!data || !result || m <= 0 || n <= 0 || k <= 0) return KMEANS_ERROR_BUILDDATA;
  if (doFullSGEMM < 0 || doFullSGEMM > 2 || matrixFormat < 0 || matrixFormat > 1)
    return KMEANS_ERROR_BUILDDATA;
  if (k > m) return KMEANS_ERROR_INITIALIZE;
  const int iters = maxIters < 0 ? 0 : maxIters;
  double sse = 0.0;
  if (initAlgorithm != KMGB_INIT_KMEANSPP)  // the reference ignores numRetries
    return run_d(data, m, n, k, criterion, iters, result, miniBatchFraction, -1, &sse);
  // k-means++ with seeds 0 .. numRetries-1; the lowest final SSE wins (the first on ties)
  const int retries = numRetries < 1 ? 1 : numRetries;
  double best_sse = std::nan("");
  kmeansErrorStatus best_st = KMEANS_SUCCESS;
  std::vector<double> tmp((size_t)n * k), keep((size_t)n * k);
  for (int r = 0; r < retries; ++r) {
    const kmeansErrorStatus st =
        run_d(data, m, n, k, criterion, iters, tmp.data(), miniBatchFraction, r, &sse);
    if (st != KMEANS_SUCCESS && st != KMEANS_NONCONVERGENCE) return st;
    if (r == 0 || sse < best_sse || (std::isnan(best_sse) && !std::isnan(sse))) {
      best_sse = sse;
      best_st = st;
      keep.swap(tmp);
    }
  }
  std::memcpy(result, keep.data(), sizeof(double) * keep.size());
  return best_st;
}
