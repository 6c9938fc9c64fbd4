// Exact re-rank of the points whose approximate top-2 margin did not certify the arg-min.
//
// Stages in this file: the candidate path of the tensor tiers (gather_flagged_kernel copies the
// flagged rows for the candidate pass; resolve_candidates_kernel settles each point from its
// recorded candidates in FP32, then float-float, then exact FP64), the tiled FP32 stage and the
// tiled exact FP64 stage for everything else, the per-point kernel described next (both modes),
// and the grouped kernel of batched problems.
//
// Per-point kernel: one warp per flagged point, lanes over centers. Pass 1 evaluates every usable center in
// FP32 together with a rigorous interval [lo_j, hi_j] around the exact value and takes
// best_hi = min_j hi_j. Pass 2 re-evaluates the centers with lo_j <= best_hi (the only ones
// that can be the FP64 arg-min) in FP64 exactly as the oracle does and keeps the smallest,
// lowest index on ties (the reference's tie rule, RowTransformMinimum.cu:43-50). A point with
// a single candidate is settled by FP32 alone; the others are counted as FP64 re-ranks.
//
// mode 0 (Lloyd):      value = sum_d (x_d - c_d)^2     FP32: fma chain of fl(x-c)^2,
//                      |err| <= ((1+u)^2 (1+gamma_D) - 1) * value (all terms non-negative).
// mode 1 (expansion):  value = nb_j - 2 x.c_j with the caller's norms nb (per-kernel ABI,
//                      KmeansCudaKernels.h:238-244); absolute bound from ||x|| and max ||c||.
#include <cfloat>
#include <cstdint>

#include <cmath>

#include "common.cuh"
#include "kernels.h"

namespace kmgb {
namespace {

__device__ __forceinline__ float approx_value(int mode, const float* __restrict__ xs,
                                              const float* __restrict__ c, int d, float nbj) {
  float a = 0.0f;
  if (mode == 0) {
    for (int t = 0; t < d; ++t) {
      const float u = xs[t] - ld(c + t);
      a = fmaf(u, u, a);
    }
    return a;
  }
  for (int t = 0; t < d; ++t) a = fmaf(xs[t], ld(c + t), a);
  return fmaf(-2.0f, a, nbj);
}

__device__ __forceinline__ double exact_value(int mode, const float* __restrict__ xs,
                                              const float* __restrict__ c, int d, float nbj) {
  double s = 0.0;
  if (mode == 0) {
    for (int t = 0; t < d; ++t) {
      const double u = (double)xs[t] - (double)ld(c + t);
      s = fma(u, u, s);
    }
    return s;
  }
  for (int t = 0; t < d; ++t) s = fma((double)xs[t], (double)ld(c + t), s);
  return fma(-2.0, s, (double)nbj);
}

__global__ void rerank_kernel(RerankArgs a) {
  if (grid_enter()) return;
  if (stopped(a.stop)) return;
  extern __shared__ float xs_all[];
  const int warps = blockDim.x >> 5;
  const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
  float* xs = xs_all + (size_t)w * a.d;
  const bool all = a.redo && pinned(a.redo) != 0;
  const long long cnt = all ? a.n : min((long long)pinned(a.count), a.max_list);
  const float u = 5.9604645e-8f;
  const float gam = (float)(a.d + 4) * 2.0f * u * 1.01f;  // mode 0 relative bound (doubled)
  for (long long slot = (long long)blockIdx.x * warps + w; slot < cnt;
       slot += (long long)gridDim.x * warps) {
    const int pt = all ? (int)slot : a.list[slot];
    const float* x = a.X + (size_t)pt * a.ldx;
    for (int t = lane; t < a.d; t += 32) xs[t] = x[t];
    __syncwarp();
    float e1 = 0.0f;
    if (a.mode == 1) {
      const float xn = a.xnorm[pt], cm = *a.cmax;
      const float gd = (float)a.d * u * 1.001f;
      e1 = (2.0f * gd * xn * cm + u * 2.01f * xn * cm +
            (float)(a.d + 2) * 2.3e-16f * xn * cm) * 1.01f;
    }
    // pass 1: best upper end
    float best_hi = INFINITY;
    for (int j = lane; j < a.k; j += 32) {
      float nbj = 0.0f;
      if (a.mode == 0) {
        if (!(a.cn[j] < INFINITY)) continue;  // unusable (empty-cluster) center
      } else {
        nbj = a.nb[j];
      }
      const float v = approx_value(a.mode, xs, a.C + (size_t)j * a.ldc, a.d, nbj);
      float hi;
      if (a.mode == 0) hi = v * (1.0f + gam) + 1e-30f;
      else hi = v + e1 + u * 1.01f * fabsf(nbj) + 1e-30f;
      if (hi < best_hi) best_hi = hi;  // NaN never passes
    }
    for (int o = 16; o > 0; o >>= 1) best_hi = fminf(best_hi, __shfl_xor_sync(0xffffffffu, best_hi, o));
    // pass 2: exact value of every candidate
    double best = INFINITY;
    int bidx = -1;
    int ncand = 0;
    for (int j = lane; j < a.k; j += 32) {
      float nbj = 0.0f;
      if (a.mode == 0) {
        if (!(a.cn[j] < INFINITY)) continue;
      } else {
        nbj = a.nb[j];
      }
      const float* c = a.C + (size_t)j * a.ldc;
      const float v = approx_value(a.mode, xs, c, a.d, nbj);
      float lo;
      if (a.mode == 0) lo = v * (1.0f - gam) - 1e-30f;
      else lo = v - e1 - u * 1.01f * fabsf(nbj) - 1e-30f;
      if (!(lo <= best_hi) && !(a.mode == 1 && lo != lo)) continue;  // (NaN: as in exact_pass)
      ++ncand;
      const double ex = exact_value(a.mode, xs, c, a.d, nbj);
      if (ex < best) {  // lanes visit their centers in increasing j: first wins ties
        best = ex;
        bidx = j;
      }
    }
    for (int o = 16; o > 0; o >>= 1) {
      const double ob = __shfl_xor_sync(0xffffffffu, best, o);
      const int oi = __shfl_xor_sync(0xffffffffu, bidx, o);
      const bool take = (ob < best) || (ob == best && (unsigned)oi < (unsigned)bidx);
      best = take ? ob : best;
      bidx = take ? oi : bidx;
      ncand += __shfl_xor_sync(0xffffffffu, ncand, o);
    }
    if (lane == 0) {
      a.labels[pt] = bidx < 0 ? 0 : bidx;
      if (a.stats) {
        atomicAdd(a.stats, 1ull);
        if (ncand > 1) atomicAdd(a.stats + 1, 1ull);
      }
    }
    __syncwarp();
  }
}

// Tiled FP32 stage of the re-rank (described for mode 0): 32 flagged points per CTA iteration against
// 64-center blocks staged in shared memory; each thread accumulates 4 points x 2 centers of
// sum_d (x_d - c_d)^2 with float4 loads. Per point (best, index, second) is merged over the 32
// threads that share it (lowest index on ties) and certified with the relative bound of the
// direct form; uncertified points go to list2 for the exact FP64 stage.
// The dynamic shared memory that launches here may ask for. Always this limit is set, not a launch's
// own size: another thread's smaller one could arrive between the call and the launch.
constexpr int kMaxTileSmem = 200 * 1024;
// From here on a launch sets it: the 48 KB that need no setting are for dynamic and static shared memory
// together, and the tiled kernels have up to 7 KB of static arrays.
constexpr size_t kPlainSmem = 40 * 1024;
constexpr int TP = 32;   // points per CTA iteration
constexpr int TC = 64;   // centers per block

// The tiled stages' two forms. A center's offset: MODE 0 zero, MODE 1 its norm; +inf for padding and
// (MODE 0) unusable centers.
template <int MODE>
__device__ __forceinline__ float tile_offset(const RerankArgs& a, int j) {
  if (j >= a.k) return INFINITY;
  if (MODE == 1) return a.nb[j];
  return a.cn[j] < INFINITY ? 0.0f : INFINITY;
}
template <int MODE>
__device__ __forceinline__ void tile_acc(const float4 x, const float4 c, float& acc) {
  if (MODE == 0) {
    float t;
    t = x.x - c.x; acc = fmaf(t, t, acc);
    t = x.y - c.y; acc = fmaf(t, t, acc);
    t = x.z - c.z; acc = fmaf(t, t, acc);
    t = x.w - c.w; acc = fmaf(t, t, acc);
  } else {
    acc = fmaf(x.x, c.x, acc);
    acc = fmaf(x.y, c.y, acc);
    acc = fmaf(x.z, c.z, acc);
    acc = fmaf(x.w, c.w, acc);
  }
}
// MODE 1: bound of |fl(nb_j - 2 x.c_j) - the FP64 value| over every center (|nb_j| <= cmax^2).
__device__ __forceinline__ float expansion_bound(const RerankArgs& a, int pt) {
  const float u = 5.9604645e-8f;
  const float xn = a.xnorm[pt], cm = *a.cmax;
  const float gd = (float)a.d * u * 1.001f;
  return (2.0f * gd * xn * cm + u * 2.01f * xn * cm + (float)(a.d + 2) * 2.3e-16f * xn * cm +
          u * 1.01f * cm * cm) * 1.01f + 1e-30f;
}

// The exact pass over the points g0 .. of a.list whose rows lie in xs (see rerank_exact_kernel): every
// (point, center) pair whose lower end is within the point's best upper end hs (NaN: a settled point,
// left alone). all: point g is row g (RerankArgs::redo).
template <int MODE, bool RECORD>
__device__ __forceinline__ void exact_pass(const RerankArgs& a, const float4* xs, float4* cs,
                                           float* cflag, int rs, int dq, long long g0, long long cnt,
                                           const float* hs, const float* es, int* __restrict__ cand,
                                           int* __restrict__ cand_cnt, bool all = false) {
  __shared__ double mb[8][TP];
  __shared__ int mi[8][TP];
  __shared__ int ncand[TP];
  const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
  const int pq = tid & 7;                 // points pq, pq + 8, pq + 16, pq + 24
  const int cq = tid >> 3;                // centers cq*2, cq*2+1 of the block
  const float u = 5.9604645e-8f;
  const float gam = (float)(a.d + 4) * 2.0f * u * 1.01f;
  if (RECORD && tid < TP) ncand[tid] = 0;
  double be[4];
  int bi[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    be[i] = INFINITY;
    bi[i] = -1;
  }
  for (int j0 = 0; j0 < a.k; j0 += TC) {
    __syncthreads();
    for (int e = tid; e < TC * dq; e += blockDim.x) {
      const int r = e / dq, q = e % dq;
      float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
      if (j0 + r < a.k) v = *reinterpret_cast<const float4*>(a.C + (size_t)(j0 + r) * a.ldc + q * 4);
      cs[r * rs + q] = v;
    }
    if (tid < TC) {
      const int j = j0 + tid;
      cflag[tid] = tile_offset<MODE>(a, j);
    }
    __syncthreads();
    float acc[4][2];
#pragma unroll
    for (int i = 0; i < 4; ++i) acc[i][0] = acc[i][1] = 0.0f;
    for (int q = 0; q < dq; ++q) {
      const float4 c0 = cs[(cq * 2) * rs + q];
      const float4 c1 = cs[(cq * 2 + 1) * rs + q];
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const float4 x = xs[(pq + 8 * i) * rs + q];
        tile_acc<MODE>(x, c0, acc[i][0]);
        tile_acc<MODE>(x, c1, acc[i][1]);
      }
    }
#pragma unroll
    for (int jj = 0; jj < 2; ++jj) {
      const int cl = cq * 2 + jj;
      const int j = j0 + cl;
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int pl = pq + 8 * i;
        // unusable (empty-cluster) or padding center
        if (MODE == 0 ? cflag[cl] != 0.0f : j >= a.k) continue;
        const float lo = MODE == 0 ? acc[i][jj] * (1.0f - gam) - 1e-30f
                                   : fmaf(-2.0f, acc[i][jj], cflag[cl]) - es[pl];
        // MODE 1: a value that overflowed FP32 under an infinite bound says nothing (inf - inf), so
        // the pair is evaluated; a settled point's NaN end still leaves it alone
        if (!(lo <= hs[pl]) && !(MODE == 1 && lo != lo && hs[pl] == hs[pl])) continue;
        if (RECORD) {
          const int at = atomicAdd(&ncand[pl], 1);
          if (at < kMaxCand) cand[(g0 + pl) * kMaxCand + at] = j;
          continue;
        }
        // FP64 in the oracle's order: dimensions 0 .. d-1 (padding dimensions are zero)
        double ex = 0.0;
        for (int q = 0; q < dq; ++q) {
          const float4 x = xs[pl * rs + q];
          const float4 c = cs[cl * rs + q];
          if (MODE == 0) {
            double dd;
            dd = (double)x.x - (double)c.x; ex = fma(dd, dd, ex);
            dd = (double)x.y - (double)c.y; ex = fma(dd, dd, ex);
            dd = (double)x.z - (double)c.z; ex = fma(dd, dd, ex);
            dd = (double)x.w - (double)c.w; ex = fma(dd, dd, ex);
          } else {
            ex = fma((double)x.x, (double)c.x, ex);
            ex = fma((double)x.y, (double)c.y, ex);
            ex = fma((double)x.z, (double)c.z, ex);
            ex = fma((double)x.w, (double)c.w, ex);
          }
        }
        if (MODE == 1) ex = fma(-2.0, ex, (double)cflag[cl]);
        if (ex < INFINITY && (ex < be[i] || (ex == be[i] && (unsigned)j < (unsigned)bi[i]))) {
          be[i] = ex;
          bi[i] = j;
        }
      }
    }
  }
  if (RECORD) {
    __syncthreads();
    if (tid < TP && g0 + tid < cnt) cand_cnt[g0 + tid] = ncand[tid] <= kMaxCand ? ncand[tid] : -1;
    return;
  }
  // merge the 32 threads of each point: lanes pq, pq+8, pq+16, pq+24 of every warp
#pragma unroll
  for (int i = 0; i < 4; ++i) {
#pragma unroll
    for (int off = 8; off < 32; off <<= 1) {
      const double ob = __shfl_xor_sync(0xffffffffu, be[i], off);
      const int oi = __shfl_xor_sync(0xffffffffu, bi[i], off);
      const bool take = (ob < be[i]) || (ob == be[i] && (unsigned)oi < (unsigned)bi[i]);
      be[i] = take ? ob : be[i];
      bi[i] = take ? oi : bi[i];
    }
    if (lane < 8) {
      mb[w][pq + 8 * i] = be[i];
      mi[w][pq + 8 * i] = bi[i];
    }
  }
  __syncthreads();
  if (tid < TP && g0 + tid < cnt && hs[tid] == hs[tid]) {
    double fb = mb[0][tid];
    int fi = mi[0][tid];
    for (int ww = 1; ww < 8; ++ww) {
      const bool take = (mb[ww][tid] < fb) || (mb[ww][tid] == fb && (unsigned)mi[ww][tid] < (unsigned)fi);
      fb = take ? mb[ww][tid] : fb;
      fi = take ? mi[ww][tid] : fi;
    }
    a.labels[all ? g0 + tid : a.list[g0 + tid]] = fi < 0 ? 0 : fi;
  }
}

template <int MODE, bool SETTLE>
__global__ void __launch_bounds__(256)
rerank_tiled_kernel(RerankArgs a, int* __restrict__ list2, int* __restrict__ count2,
                    float* __restrict__ hi2) {
  if (grid_enter()) return;
  const int halt = a.stop ? pinned(a.stop) : 0;
  const bool all = MODE == 1 && SETTLE && a.redo && pinned(a.redo) != 0;
  const long long cnt = all ? a.n : min((long long)pinned(a.count), a.max_list);
  if (halt) return;
  extern __shared__ float4 sm4[];
  const int dq = (a.d + 3) >> 2;          // float4 per row
  const int rs = (dq + 1) | 1;            // row stride in float4, odd: 8 consecutive rows' columns
                                          // lie in distinct banks
  float4* xs = sm4;                       // [TP][rs]
  float4* cs = xs + TP * rs;              // [TC][rs]
  float* cflag = reinterpret_cast<float*>(cs + TC * rs);  // [TC] value offset (tile_offset)
  __shared__ float mb1[8][TP], mb2[8][TP];
  __shared__ int mi1[8][TP];
  __shared__ float hs[TP], es[TP];
  const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
  const int pq = tid & 7;                 // points pq, pq + 8, pq + 16, pq + 24
  const int cq = tid >> 3;                // centers cq*2, cq*2+1 of the block
  if (a.counts && a.stats && blockIdx.x == 0 && tid == 0) {
    a.stats[0] += (unsigned long long)a.counts[0];
    a.stats[1] += (unsigned long long)a.counts[a.full_idx];
  }
  const float u = 5.9604645e-8f;
  const float gam = (float)(a.d + 4) * 2.0f * u * 1.01f;

  for (long long g0 = (long long)blockIdx.x * TP; g0 < cnt; g0 += (long long)gridDim.x * TP) {
    __syncthreads();
    // stage the points (zero rows past the list end)
    for (int e = tid; e < TP * dq; e += blockDim.x) {
      const int r = e / dq, q = e % dq;
      float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
      if (g0 + r < cnt) {
        const float* x = a.X + (size_t)(all ? g0 + r : a.list[g0 + r]) * a.ldx;
        const int c0 = q * 4;
        v.x = c0 < a.d ? x[c0] : 0.f;
        v.y = c0 + 1 < a.d ? x[c0 + 1] : 0.f;
        v.z = c0 + 2 < a.d ? x[c0 + 2] : 0.f;
        v.w = c0 + 3 < a.d ? x[c0 + 3] : 0.f;
      }
      xs[r * rs + q] = v;
    }
    float b1[4], b2[4];
    int i1[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      b1[i] = INFINITY;
      b2[i] = INFINITY;
      i1[i] = -1;
    }
    for (int j0 = 0; j0 < a.k; j0 += TC) {
      __syncthreads();
      for (int e = tid; e < TC * dq; e += blockDim.x) {
        const int r = e / dq, q = e % dq;
        float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
        if (j0 + r < a.k) {
          const float* c = a.C + (size_t)(j0 + r) * a.ldc;
          const int c0 = q * 4;  // ldc is a multiple of 4 and rows are zero padded
          v = *reinterpret_cast<const float4*>(c + c0);
        }
        cs[r * rs + q] = v;
      }
      if (tid < TC) {
        const int j = j0 + tid;
        cflag[tid] = tile_offset<MODE>(a, j);
      }
      __syncthreads();
      float acc[4][2];
#pragma unroll
      for (int i = 0; i < 4; ++i) acc[i][0] = acc[i][1] = 0.0f;
      for (int q = 0; q < dq; ++q) {
        const float4 c0 = cs[(cq * 2) * rs + q];
        const float4 c1 = cs[(cq * 2 + 1) * rs + q];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const float4 x = xs[(pq + 8 * i) * rs + q];
          tile_acc<MODE>(x, c0, acc[i][0]);
          tile_acc<MODE>(x, c1, acc[i][1]);
        }
      }
#pragma unroll
      for (int jj = 0; jj < 2; ++jj) {
        const int j = j0 + cq * 2 + jj;
        const float f = cflag[cq * 2 + jj];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          // +inf for unusable / padding centers
          const float v = MODE == 0 ? acc[i][jj] + f : fmaf(-2.0f, acc[i][jj], f);
          const float nb2 = fminf(b2[i], fmaxf(b1[i], v));
          const bool lt = v < b1[i];
          b1[i] = lt ? v : b1[i];
          i1[i] = lt ? j : i1[i];
          b2[i] = nb2;
        }
      }
    }
    // merge the 32 threads of each point: lanes pq, pq+8, pq+16, pq+24 of every warp
#pragma unroll
    for (int i = 0; i < 4; ++i) {
#pragma unroll
      for (int off = 8; off < 32; off <<= 1) {
        const float ob1 = __shfl_xor_sync(0xffffffffu, b1[i], off);
        const float ob2 = __shfl_xor_sync(0xffffffffu, b2[i], off);
        const int oi1 = __shfl_xor_sync(0xffffffffu, i1[i], off);
        const float nb2 = fminf(fminf(b2[i], ob2), fmaxf(b1[i], ob1));
        const bool take = (ob1 < b1[i]) || (ob1 == b1[i] && (unsigned)oi1 < (unsigned)i1[i]);
        b1[i] = take ? ob1 : b1[i];
        i1[i] = take ? oi1 : i1[i];
        b2[i] = nb2;
      }
      if (lane < 8) {
        mb1[w][pq + 8 * i] = b1[i];
        mb2[w][pq + 8 * i] = b2[i];
        mi1[w][pq + 8 * i] = i1[i];
      }
    }
    __syncthreads();
    if (tid < TP && g0 + tid < cnt) {
      float f1 = mb1[0][tid], f2 = mb2[0][tid];
      int fi = mi1[0][tid];
      for (int ww = 1; ww < 8; ++ww) {
        const float ob1 = mb1[ww][tid], ob2 = mb2[ww][tid];
        const int oi1 = mi1[ww][tid];
        const float nb2 = fminf(fminf(f2, ob2), fmaxf(f1, ob1));
        const bool take = (ob1 < f1) || (ob1 == f1 && (unsigned)oi1 < (unsigned)fi);
        f1 = take ? ob1 : f1;
        fi = take ? oi1 : fi;
        f2 = nb2;
      }
      const int pt = all ? (int)(g0 + tid) : a.list[g0 + tid];
      // certified when every other center's lower end exceeds the best's upper end
      float lo2, hi1;
      if (MODE == 0) {
        lo2 = f2 * (1.0f - gam) - 1e-30f;
        hi1 = f1 * (1.0f + gam) + 1e-30f;  // no usable center: +inf
      } else {
        const float e = expansion_bound(a, pt);
        lo2 = f2 - e;
        hi1 = f1 + e;
        if (!(hi1 == hi1)) hi1 = INFINITY;
      }
      const bool settled = fi >= 0 && lo2 > hi1;
      if (settled) a.labels[pt] = fi;
      if (SETTLE) {
        hs[tid] = settled ? __int_as_float(0x7fc00000) : hi1;
        es[tid] = MODE == 1 ? expansion_bound(a, pt) : 0.0f;
      } else if (!settled) {
        const int slot = atomicAdd(count2, 1);
        list2[slot] = pt;
        hi2[slot] = hi1;
      }
    } else if (SETTLE && tid < TP) {
      hs[tid] = __int_as_float(0x7fc00000);
      es[tid] = 0.0f;
    }
    if (SETTLE && __syncthreads_or(tid < TP && hs[tid] == hs[tid]))
      exact_pass<MODE, false>(a, xs, cs, cflag, rs, dq, g0, cnt, hs, es, nullptr, nullptr, all);
  }
}

// Exact stage of the Lloyd re-rank (mode 0), tiled like the FP32 stage: 32 residual points per
// CTA iteration against 64-center blocks staged in shared memory. Every (point, usable center)
// pair whose FP32 direct-form lower end is within the point's best upper end (hi2, from the FP32
// stage) is evaluated in FP64 in the oracle's order (sequential fma over the dimensions); the
// smallest value wins, lowest index on ties. Centers are read once per 32 points, so the cost
// stays that of one tiled FP32 scan however many points reach this stage.
//
// RECORD: instead of evaluating the pairs inside the band in FP64 (where one thread's evaluation
// holds its whole warp on the narrow FP64 pipe), the band's centers become the candidates of
// resolve_candidates_kernel, whose float-float tier settles nearly all of them: 796,160 x 324,
// K=256, FP32 tier, 1.05 ms per iteration before. Slots from cand_cap on go to over / over_hi.
template <bool RECORD>
__global__ void __launch_bounds__(256)
rerank_exact_kernel(RerankArgs a, const float* hi2, int* __restrict__ cand,
                    int* __restrict__ cand_cnt, long long cand_cap, int* __restrict__ over,
                    int* __restrict__ over_count, float* __restrict__ over_hi) {
  if (grid_enter()) return;
  if (stopped(a.stop)) return;
  extern __shared__ float4 sm4[];
  const int dq = (a.d + 3) >> 2;
  const int rs = (dq + 1) | 1;
  float4* xs = sm4;                       // [TP][rs]
  float4* cs = xs + TP * rs;              // [TC][rs]
  float* cflag = reinterpret_cast<float*>(cs + TC * rs);  // [TC] value offset (tile_offset)
  __shared__ float hs[TP];
  const int tid = threadIdx.x;
  long long cnt = min((long long)pinned(a.count), a.max_list);
  if (RECORD && cnt > cand_cap) {
    for (long long slot = cand_cap + (long long)blockIdx.x * blockDim.x + tid; slot < cnt;
         slot += (long long)gridDim.x * blockDim.x) {
      const int o = atomicAdd(over_count, 1);
      over[o] = a.list[slot];
      over_hi[o] = hi2[slot];
    }
    cnt = cand_cap;
  }
  for (long long g0 = (long long)blockIdx.x * TP; g0 < cnt; g0 += (long long)gridDim.x * TP) {
    __syncthreads();
    for (int e = tid; e < TP * dq; e += blockDim.x) {
      const int r = e / dq, q = e % dq;
      float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
      if (g0 + r < cnt) {
        const float* x = a.X + (size_t)a.list[g0 + r] * a.ldx;
        const int c0 = q * 4;
        v.x = c0 < a.d ? x[c0] : 0.f;
        v.y = c0 + 1 < a.d ? x[c0 + 1] : 0.f;
        v.z = c0 + 2 < a.d ? x[c0 + 2] : 0.f;
        v.w = c0 + 3 < a.d ? x[c0 + 3] : 0.f;
      }
      xs[r * rs + q] = v;
    }
    if (tid < TP) hs[tid] = (g0 + tid < cnt) ? hi2[g0 + tid] : -INFINITY;
    __syncthreads();
    exact_pass<0, RECORD>(a, xs, cs, cflag, rs, dq, g0, cnt, hs, nullptr, cand, cand_cnt);
  }
}

// Grouped (batched Lloyd) re-rank, one warp per flagged row of any problem; the row's own
// problem (tile_prob[row / 128]) gives its center range. Pass 1, FP32 direct form: L lanes split a
// center's dimensions, 16 bytes each at a time, 32 / L centers side by side and four in turn (a tree
// sum per center -- like any order it stays within the (d+4) 2u relative bound of a sum of
// non-negative terms); the values of up to RG_VCAP centers stay in shared memory. (A whole warp per
// center left 16 of 32 lanes idle at D = 16 and took four centers a step.) Pass 2: every usable center
// whose FP32 lower end is within the smallest upper end is evaluated in FP64 in the oracle's order
// (sequential fma over the dimensions), the smallest value winning, lowest index on ties.
// Labels are global center indices.
constexpr int RG_VCAP = 512;
constexpr int RG_WARPS = 8;

template <int L>
__global__ void __launch_bounds__(RG_WARPS * 32)
rerank_grouped_kernel(RerankArgs a, GroupArgs g, int* __restrict__ cand, int* __restrict__ cand_cnt,
                      long long cand_cap) {
  if (grid_enter()) return;
  if (stopped(a.stop)) return;
  extern __shared__ float rg_smem[];  // [warps][RG_VCAP] values, then [warps][ds] rows
  constexpr int G = 32 / L;           // centers side by side
  constexpr int U = 4;                // and in turn, their loads in flight together
  const long long cnt = min((long long)pinned(a.count), a.max_list);
  const float u = 5.9604645e-8f;
  const float gam = (float)(a.d + 4) * 2.0f * u * 1.01f;
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int grp = lane / L, sub = lane % L;
  const int ds = (a.d + 3) / 4 * 4;
  float* vals = rg_smem + (size_t)w * RG_VCAP;
  float* xs = rg_smem + (size_t)RG_WARPS * RG_VCAP + (size_t)w * ds;
  for (long long slot = (long long)blockIdx.x * RG_WARPS + w; slot < cnt;
       slot += (long long)gridDim.x * RG_WARPS) {
    const int pt = a.list[slot];
    const int prob = g.tile_prob[pt >> 7];
    const int cbeg = g.c_off[prob], kp = g.k[prob];
    const bool keep = kp <= RG_VCAP;
    const float* x = a.X + (size_t)pt * a.ldx;
    __syncwarp();
    for (int t = lane; t < ds; t += 32) xs[t] = t < a.d ? x[t] : 0.0f;
    __syncwarp();
    float lo = INFINITY;
    for (int j0 = 0; j0 < kp; j0 += G * U) {
      float sv[U];
      const float* cr[U];
#pragma unroll
      for (int r = 0; r < U; ++r) {
        sv[r] = 0.0f;
        cr[r] = a.C + (size_t)(cbeg + min(j0 + r * G + grp, kp - 1)) * a.ldc;
      }
      // rows are padded with zeros to ldc, a multiple of 4, as xs to ds
      for (int t = 4 * sub; t < ds; t += 4 * L) {
        const float4 xt = *reinterpret_cast<const float4*>(xs + t);
#pragma unroll
        for (int r = 0; r < U; ++r) tile_acc<0>(xt, ld(reinterpret_cast<const float4*>(cr[r] + t)), sv[r]);
      }
#pragma unroll
      for (int o = L / 2; o > 0; o >>= 1) {
#pragma unroll
        for (int r = 0; r < U; ++r) sv[r] += __shfl_xor_sync(0xffffffffu, sv[r], o);
      }
#pragma unroll
      for (int r = 0; r < U; ++r) {
        const int j = j0 + r * G + grp;
        if (j < kp) {
          const float v = (a.cn[cbeg + j] < INFINITY) ? sv[r] : INFINITY;  // unusable center
          lo = fminf(lo, v);
          if (keep && sub == 0) vals[j] = v;
        }
      }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) lo = fminf(lo, __shfl_xor_sync(0xffffffffu, lo, o));
    __syncwarp();
    const float best_hi = lo * (1.0f + gam) + 1e-30f;
    if (cand && slot < cand_cap) {
      // record the band (every center whose FP64 distance can be the minimum) for the
      // candidate resolve's FP32 and float-float tiers; more than kMaxCand: the exact pass
      int n_in = 0;
      for (int j0 = 0; j0 < kp; j0 += 32) {
        const int j = j0 + lane;
        bool in = false;
        if (j < kp && a.cn[cbeg + j] < INFINITY) {
          const float v = keep ? vals[j] : approx_value(0, xs, a.C + (size_t)(cbeg + j) * a.ldc,
                                                        a.d, 0.0f);
          in = v * (1.0f - gam) - 1e-30f <= best_hi;
        }
        const unsigned bal = __ballot_sync(0xffffffffu, in);
        const int at = n_in + __popc(bal & ((1u << lane) - 1u));
        if (in && at < kMaxCand) cand[slot * kMaxCand + at] = cbeg + j;
        n_in += __popc(bal);
      }
      if (lane == 0) {
        cand_cnt[slot] = n_in <= kMaxCand ? n_in : -1;
        if (a.stats) atomicAdd(a.stats, 1ull);
      }
      continue;
    }
    double best = INFINITY;
    int bidx = -1;
    for (int j = lane; j < kp; j += 32) {
      if (!(a.cn[cbeg + j] < INFINITY)) continue;
      const float* c = a.C + (size_t)(cbeg + j) * a.ldc;
      const float v = keep ? vals[j] : approx_value(0, xs, c, a.d, 0.0f);
      if (!(v * (1.0f - gam) - 1e-30f <= best_hi)) continue;
      const double ex = exact_value(0, xs, c, a.d, 0.0f);
      if (ex < best) {  // a lane's centers come in increasing index order
        best = ex;
        bidx = j;
      }
    }
    for (int o = 16; o > 0; o >>= 1) {
      const double ob = __shfl_xor_sync(0xffffffffu, best, o);
      const int oi = __shfl_xor_sync(0xffffffffu, bidx, o);
      const bool take = (ob < best) || (ob == best && (unsigned)oi < (unsigned)bidx);
      best = take ? ob : best;
      bidx = take ? oi : bidx;
    }
    if (lane == 0) {
      a.labels[pt] = cbeg + (bidx < 0 ? 0 : bidx);
      if (a.stats) atomicAdd(a.stats, 1ull);
    }
  }
}

}  // namespace

namespace {
// Copies the BF16 rows (and residual rows) of the flagged points into a compact buffer, row
// `slot` for list[slot], with the point's candidate floor. The compact buffer holds `cap` rows;
// flagged points beyond it go straight to `over` (the full rescan), so any number of flagged points
// is settled exactly.
__global__ void __launch_bounds__(256, 4)
gather_flagged_kernel(const int* list, const int* count,
                                      long long cap, const uint4* Xb,
                                      const uint4* Xl, long long row_vec,
                                      const float* thr, uint4* __restrict__ XbC,
                                      uint4* __restrict__ XlC, float* __restrict__ thrC,
                                      int* __restrict__ over, int* __restrict__ over_count,
                                      const int* stop, const float* xs,
                                      float* __restrict__ xsC) {
  if (grid_enter()) return;
  const int halt = stop ? pinned(stop) : 0;
  const long long total = pinned(count);
  if (halt) return;
  const long long cnt = min(total, cap);
  const long long t0 = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  const long long nt = (long long)gridDim.x * blockDim.x;
  for (long long slot = cap + t0; slot < total; slot += nt) over[atomicAdd(over_count, 1)] = list[slot];
  for (long long slot = nt - 1 - t0; slot < cnt; slot += nt) {  // (the grid's end, while its first warps copy)
    const long long pt = list[slot];
    // without a finite floor (no usable center, an infinite bound) the keys say nothing: no key
    // reaches NaN (an infinite one would reach infinity), so no candidates, hence the full rescan
    const float fl = thr[pt];
    thrC[slot] = fl > -3.0e38f ? fl : __int_as_float(0x7fc00000);
    if (xs) xsC[slot] = xs[pt];
  }
  copy_listed_rows(list, cnt, Xb, Xl, (int)row_vec, XbC, XlC, t0 >> 5, nt >> 5, threadIdx.x & 31);
}

// Error-free float-float helpers (FP32 pipe). two_sum: s + e == a + b exactly.
__device__ __forceinline__ void two_sum(float a, float b, float& s, float& e) {
  s = __fadd_rn(a, b);
  const float bp = __fsub_rn(s, a);
  e = __fadd_rn(__fsub_rn(a, __fsub_rn(s, bp)), __fsub_rn(b, bp));
}

constexpr int kGroupLanes = 8;  // lanes per candidate in the fast path: 4 candidates at a time
static_assert(kMaxCand <= 32, "one lane per recorded candidate");

// One term of ||x - c||^2 into the float-float (hi, lo): u = x - c is split exactly into uh + ul
// (two_sum), uh^2 = p + e exactly (FMA), and the remaining 2*uh*ul + ul^2 + e is added with one
// rounding; hi collects the p's by two_sum, lo the rest.
__device__ __forceinline__ void ff_term(float xv, float cv, float& hi, float& lo) {
  float uh, ul;
  two_sum(xv, -cv, uh, ul);
  const float p = __fmul_rn(uh, uh);
  const float e = __fmaf_rn(uh, uh, -p);
  const float r = __fmaf_rn(ul, ul, __fmaf_rn(__fadd_rn(uh, uh), ul, e));
  float s, err;
  two_sum(hi, p, s, err);
  hi = s;
  lo = __fadd_rn(lo, __fadd_rn(err, r));
}

// ||x - c||^2 over the first d dimensions as a float-float (hi, lo), summed over each group of
// 8 consecutive lanes (every lane of a group ends with its group's total; all 32 lanes call it,
// a group with nothing to do passes d = 0). Lane r of a group takes dimensions 4r..4r+3,
// 4r+32.. with 16-byte loads (VEC: d, both row strides and both bases multiples of 4 floats),
// else r, r+8, ...: at most m = 4 ceil(d/32) terms per lane, then three reduction levels.
template <bool VEC>
__device__ __forceinline__ void ff_dist8(const float* __restrict__ x, const float* __restrict__ c,
                                         int d, int r, float& hi, float& lo) {
  hi = 0.0f;
  lo = 0.0f;
  if (VEC) {
    for (int t = 4 * r; t < d; t += 4 * kGroupLanes) {
      const float4 xv = ld(reinterpret_cast<const float4*>(x + t));
      const float4 cv = ld(reinterpret_cast<const float4*>(c + t));
      ff_term(xv.x, cv.x, hi, lo);
      ff_term(xv.y, cv.y, hi, lo);
      ff_term(xv.z, cv.z, hi, lo);
      ff_term(xv.w, cv.w, hi, lo);
    }
  } else {
    for (int t = r; t < d; t += kGroupLanes) ff_term(ld(x + t), ld(c + t), hi, lo);
  }
  for (int o = kGroupLanes / 2; o > 0; o >>= 1) {
    const float oh = __shfl_xor_sync(0xffffffffu, hi, o);
    const float ol = __shfl_xor_sync(0xffffffffu, lo, o);
    float s, err;
    two_sum(hi, oh, s, err);
    hi = s;
    lo = __fadd_rn(lo, __fadd_rn(ol, err));
  }
}

// ||x - c||^2 over the first d dimensions in FP32, summed over each group of 8 consecutive lanes
// (all 32 lanes call it; a group with nothing to do passes d = 0). Every step is one explicitly
// rounded operation: u = x - c, then s = u*u + s by FMA. VEC: four independent chains per lane
// (the float4 components, at most ceil(d/32) terms each) merged in two levels, then three
// butterfly levels; scalar: one chain of at most ceil(d/8) terms, then three levels.
template <bool VEC>
__device__ __forceinline__ float f32_dist8(const float* __restrict__ x, const float* __restrict__ c,
                                           int d, int r) {
  float s;
  if (VEC) {
    float a0 = 0.0f, a1 = 0.0f, a2 = 0.0f, a3 = 0.0f;
    for (int t = 4 * r; t < d; t += 4 * kGroupLanes) {
      const float4 xv = ld(reinterpret_cast<const float4*>(x + t));
      const float4 cv = ld(reinterpret_cast<const float4*>(c + t));
      const float u0 = __fsub_rn(xv.x, cv.x), u1 = __fsub_rn(xv.y, cv.y);
      const float u2 = __fsub_rn(xv.z, cv.z), u3 = __fsub_rn(xv.w, cv.w);
      a0 = __fmaf_rn(u0, u0, a0);
      a1 = __fmaf_rn(u1, u1, a1);
      a2 = __fmaf_rn(u2, u2, a2);
      a3 = __fmaf_rn(u3, u3, a3);
    }
    s = __fadd_rn(__fadd_rn(a0, a1), __fadd_rn(a2, a3));
  } else {
    s = 0.0f;
    for (int t = r; t < d; t += kGroupLanes) {
      const float u = __fsub_rn(ld(x + t), ld(c + t));
      s = __fmaf_rn(u, u, s);
    }
  }
  for (int o = kGroupLanes / 2; o > 0; o >>= 1)
    s = __fadd_rn(s, __shfl_xor_sync(0xffffffffu, s, o));
  return s;
}

// Resolves every flagged point from its recorded candidates. The candidate set holds every center
// whose FP64 distance can be the minimum; the label is the oracle's: smallest FP64 distance
// (sequential fma over the dimensions), lowest index on ties.
//
// First tier (FP32, 8 lanes per candidate, 4 candidates at a time): every term of the FP32 value
// is non-negative and passes through at most m + 7 roundings of 2^-24 (the subtraction twice, as
// u^2, then at most m = ceil(d/8) FMAs, two merges and three butterfly levels), so it is within
// rel32 = (m + 8) 2^-24 (x1.1) of the exact distance, plus abs32 for results in the subnormal
// range; with the oracle's own (d+2) 2^-52, a best candidate ahead of the runner-up by more than
// both is the oracle's arg-min. Flagged points are mostly ahead by far more than that.
//
// Second tier (FP32 pipe, 8 lanes per candidate, 4 candidates at a time): the float-float distance
// v of each candidate is within rel*v + abs of the exact distance, and the oracle's FP64 value is
// within (d+2)*2^-52 relative of it. Per lane (m = 4 ceil(d/32) terms) the lo accumulator's
// roundings are bounded by (m+1)^2 * 2^-47 relative, the 2*uh*ul + ul^2 + e terms by 2^-46, the
// three reduction levels by 3 * (m+6) * 2^-47; rel takes 8x that sum. abs covers products that
// reach the subnormal range. If the best candidate beats the runner-up by more than both
// tolerances, it is the oracle's arg-min. Otherwise (near ties, duplicate centers, non-finite
// values) the point's candidates are evaluated exactly as the oracle does, one lane per
// candidate, in FP64. Points with more candidates than recorded (or none) go to `over` for the
// full re-rank.
// The tolerances, computed on the host, the first tier's as FP32 numbers rounded up: GB300's FP64 pipe
// takes a warp 16 cycles an instruction. Twenty of them per warp of the grid, most of which find no
// point, and as many per point in the first tier were the kernel's time (1M x 256, K=16,384: 172 us an
// iteration).
struct ResolveTol {
  double rel, abs_tol;
  float rel32, twice_abs32;
};
ResolveTol resolve_tolerances(int d) {
  const double m = 4.0 * (double)((d + 31) / 32);
  const double m32 = (double)((d + kGroupLanes - 1) / kGroupLanes);
  ResolveTol t;
  t.rel = 8.0 * ((m + 1.0) * (m + 1.0) + 2.0 + 3.0 * (m + 6.0)) * 0x1p-47 + (double)(d + 2) * 0x1p-52;
  t.abs_tol = (double)(d + 32) * 0x1p-118;
  const double rel32 = 1.1 * (m32 + 8.0) * 0x1p-24 + (double)(d + 2) * 0x1p-52;
  const double abs32 = (double)(d + 32) * (m32 + 8.0) * 0x1p-149;
  t.rel32 = std::nextafter((float)rel32, INFINITY);
  t.twice_abs32 = std::nextafter((float)(2.0 * abs32), INFINITY);
  return t;
}

template <bool VEC>
__global__ void resolve_candidates_kernel(const int* list, const int* count,
                                          long long max_list, const int* cand,
                                          const int* cand_cnt,
                                          const float* X, long long ldx,
                                          const float* C, long long ldc,
                                          const float* cn, int d,
                                          int* __restrict__ labels, int* __restrict__ over,
                                          int* __restrict__ over_count, const int* stop,
                                          const int* row_map,
                                          const float* hi_in,
                                          float* __restrict__ over_hi, ResolveTol tol) {
  if (grid_enter()) return;
  const int halt = stop ? pinned(stop) : 0;
  const long long cnt = min((long long)pinned(count), max_list);
  if (halt || cnt <= 0) return;
  const int lane = threadIdx.x & 31;
  const int grp = lane / kGroupLanes, sub = lane % kGroupLanes;
  constexpr int kGroups = 32 / kGroupLanes;
  const long long w0 = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const long long nw = ((long long)gridDim.x * blockDim.x) >> 5;
  // a point this kernel cannot settle, with its band's upper end where the list carries them
  auto to_over = [&](int pt, long long slot) {
    const int o = atomicAdd(over_count, 1);
    over[o] = pt;
    if (over_hi) over_hi[o] = hi_in[slot];
  };
  for (long long slot = w0; slot < cnt; slot += nw) {
    const int pt = list[slot];
    // with row_map (routed scan) the candidates are kept per routed row pt, and the point's FP32
    // row is row_map[pt]; otherwise per list slot, and the row is pt
    const long long ci = row_map ? (long long)pt : slot;
    const int nc = cand_cnt[ci];
    if (nc <= 0 || nc > kMaxCand) {
      if (lane == 0) to_over(pt, slot);
      continue;
    }
    const float* x = X + (size_t)(row_map ? row_map[pt] : pt) * ldx;
    // lane q holds candidate q and whether it is usable
    const int myj = lane < nc ? cand[ci * kMaxCand + lane] : -1;
    const int myok = (myj >= 0 && cn[myj] < INFINITY) ? 1 : 0;
    // both fast tiers certify only a strict separation, so the list order (column slice by
    // column slice) does not matter. First tier: lane q ends with candidate q's value; values are
    // non-negative, so their bits order as they do
    float mv = INFINITY;
    for (int q0 = 0; q0 < nc; q0 += kGroups) {
      const int q = q0 + grp;  // <= 31: q0 is a multiple of 4 below nc <= kMaxCand = 32
      const int j = __shfl_sync(0xffffffffu, myj, q);
      const int ok = __shfl_sync(0xffffffffu, myok, q) && q < nc;
      const float v = f32_dist8<VEC>(x, ok ? C + (size_t)j * ldc : x, ok ? d : 0, sub);
      const float vq = __shfl_sync(0xffffffffu, v, (lane - q0) % kGroups * kGroupLanes);
      if (lane >= q0 && lane < q0 + kGroups) mv = vq;
    }
    if (!__any_sync(0xffffffffu, myok)) {  // no usable candidate
      if (lane == 0) to_over(pt, slot);
      continue;
    }
    bool finite = !__any_sync(0xffffffffu, myok && !(mv < 3.0e38f));  // overflow, inf or NaN
    const unsigned bits = __float_as_uint(myok && finite ? mv : INFINITY);
    const unsigned b1 = __reduce_min_sync(0xffffffffu, bits);
    const int at = __ffs(__ballot_sync(0xffffffffu, bits == b1)) - 1;
    const unsigned b2 = __reduce_min_sync(0xffffffffu, lane == at ? 0x7f800000u : bits);
    // one usable candidate (the second infinite, its own value finite) is the arg-min itself
    const float f1 = __uint_as_float(b1), f2 = __uint_as_float(b2);
    if (finite &&
        (f2 == INFINITY ||
         __fsub_rd(f2, f1) > __fmaf_ru(__fadd_ru(f1, f2), tol.rel32, tol.twice_abs32))) {
      if (lane == at) labels[pt] = myj;
      continue;
    }
    double v1 = INFINITY, v2 = INFINITY;
    int i1 = -1;
    finite = true;
    for (int q0 = 0; q0 < nc; q0 += kGroups) {
      const int q = q0 + grp;  // <= 31: q0 is a multiple of 4 below nc <= kMaxCand = 32
      const int j = __shfl_sync(0xffffffffu, myj, q);
      const int ok = __shfl_sync(0xffffffffu, myok, q) && q < nc;
      float hi, lo;
      ff_dist8<VEC>(x, ok ? C + (size_t)j * ldc : x, ok ? d : 0, sub, hi, lo);
      const double v = (double)hi + (double)lo;
      for (int g = 0; g < kGroups; ++g) {
        const double vg = __shfl_sync(0xffffffffu, v, g * kGroupLanes);
        const int jg = __shfl_sync(0xffffffffu, j, g * kGroupLanes);
        if (!__shfl_sync(0xffffffffu, ok, g * kGroupLanes)) continue;
        if (!(vg < 1.0e300)) finite = false;  // overflow, inf or NaN on the FP32 pipe
        if (vg < v1) {
          v2 = v1;
          v1 = vg;
          i1 = jg;
        } else if (vg < v2) {
          v2 = vg;
        }
      }
    }
    if (i1 < 0) {  // no usable candidate
      if (lane == 0) to_over(pt, slot);
      continue;
    }
    // one usable candidate (v2 infinite, every value finite) is the arg-min itself; the
    // comparison below would read inf > inf
    if (finite && (v2 == INFINITY || v2 - v1 > (v1 + v2) * tol.rel + 2.0 * tol.abs_tol)) {
      if (lane == 0) labels[pt] = i1;
      continue;
    }
    // exact path: the oracle's sequential FP64 evaluation, lane l taking candidates l, l+32, ...;
    // equal values go to the lowest center index, within a lane and across lanes
    double best = INFINITY;
    int bidx = -1;
    for (int q = lane; q < nc; q += 32) {
      const int j = cand[ci * kMaxCand + q];
      if (cn[j] < INFINITY) {
        const float* c = C + (size_t)j * ldc;
        double s = 0.0;
        for (int t = 0; t < d; ++t) {
          const double u = (double)ld(x + t) - (double)ld(c + t);
          s = fma(u, u, s);
        }
        if (s < INFINITY && (s < best || (s == best && (unsigned)j < (unsigned)bidx))) {
          best = s;  // the oracle never takes a NaN or infinite distance
          bidx = j;
        }
      }
    }
    for (int o = 16; o > 0; o >>= 1) {
      const double ob = __shfl_xor_sync(0xffffffffu, best, o);
      const int oi = __shfl_xor_sync(0xffffffffu, bidx, o);
      const bool take = (ob < best) || (ob == best && (unsigned)oi < (unsigned)bidx);
      best = take ? ob : best;
      bidx = take ? oi : bidx;
    }
    if (lane == 0) {
      if (bidx < 0) to_over(pt, slot);
      else labels[pt] = bidx;
    }
  }
}

// x.c over the first d dimensions as a float-float (hi, lo), summed over each group of 8 consecutive
// lanes as in ff_dist8: exact products (p + e by FMA), TwoSum.
__device__ __forceinline__ void ff_product(float x, float c, float& hi, float& lo) {
  const float p = __fmul_rn(x, c);
  const float e = __fmaf_rn(x, c, -p);
  float s, err;
  two_sum(hi, p, s, err);
  hi = s;
  lo = __fadd_rn(lo, __fadd_rn(err, e));
}
template <bool VEC>
__device__ __forceinline__ void ff_dot8(const float* __restrict__ x, const float* __restrict__ c, int d,
                                        int r, float& hi, float& lo) {
  hi = 0.0f;
  lo = 0.0f;
  if (VEC) {
    for (int t = 4 * r; t < d; t += 4 * kGroupLanes) {
      const float4 xv = ld(reinterpret_cast<const float4*>(x + t));
      const float4 cv = ld(reinterpret_cast<const float4*>(c + t));
      ff_product(xv.x, cv.x, hi, lo);
      ff_product(xv.y, cv.y, hi, lo);
      ff_product(xv.z, cv.z, hi, lo);
      ff_product(xv.w, cv.w, hi, lo);
    }
  } else {
    for (int t = r; t < d; t += kGroupLanes) ff_product(ld(x + t), ld(c + t), hi, lo);
  }
  for (int o = kGroupLanes / 2; o > 0; o >>= 1) {
    const float oh = __shfl_xor_sync(0xffffffffu, hi, o);
    const float ol = __shfl_xor_sync(0xffffffffu, lo, o);
    float s, err;
    two_sum(hi, oh, s, err);
    hi = s;
    lo = __fadd_rn(lo, __fadd_rn(ol, err));
  }
}

// Expansion form (mode 1, value nb_j - 2 x.c_j): the recorded candidates of every flagged point in
// float-float, eight lanes per candidate. Each dot product is within rel sum|x_t c_t| <= rel ||x||
// cmax of the exact one (rel: resolve_candidates_kernel's, for products instead of squares) and the
// FP64 value the label is defined by within (d + 4) 2^-52 (||x|| + cmax)^2; a best candidate ahead by
// more than both, twice, is the arg-min. Other points (ties, non-finite values) take the sequential
// FP64 evaluation, one lane per candidate, lowest index on ties.
template <bool VEC>
__global__ void resolve_expansion_kernel(RerankArgs a, const int* cand,
                                         const int* cand_cnt, int* __restrict__ over,
                                         int* __restrict__ over_count) {
  if (grid_enter()) return;
  const long long cnt = min((long long)pinned(a.count), a.max_list);
  const int lane = threadIdx.x & 31;
  const int grp = lane / kGroupLanes, sub = lane % kGroupLanes;
  constexpr int kGroups = 32 / kGroupLanes;
  const long long w0 = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const long long nw = ((long long)gridDim.x * blockDim.x) >> 5;
  const int d = a.d;
  const double m = 4.0 * (double)((d + 31) / 32);
  const double rel = 8.0 * ((m + 1.0) * (m + 1.0) + 2.0 + 3.0 * (m + 6.0)) * 0x1p-47;
  const double cm = (double)*a.cmax;
  for (long long slot = w0; slot < cnt; slot += nw) {
    const int pt = a.list[slot];
    const int nc = cand_cnt[slot];
    if (nc <= 0 || nc > kMaxCand) {
      if (lane == 0) over[atomicAdd(over_count, 1)] = pt;
      continue;
    }
    const float* x = a.X + (size_t)pt * a.ldx;
    const int myj = lane < nc ? cand[slot * kMaxCand + lane] : -1;
    const float mynb = myj >= 0 && myj < a.k ? a.nb[myj] : INFINITY;
    const int myok = mynb < INFINITY ? 1 : 0;  // a NaN or infinite norm never wins
    double v1 = INFINITY, v2 = INFINITY;
    int i1 = -1;
    bool finite = true;
    for (int q0 = 0; q0 < nc; q0 += kGroups) {
      const int q = q0 + grp;
      const int j = __shfl_sync(0xffffffffu, myj, q);
      const int ok = __shfl_sync(0xffffffffu, myok, q) && q < nc;
      const float nbj = __shfl_sync(0xffffffffu, mynb, q);
      float hi, lo;
      ff_dot8<VEC>(x, ok ? a.C + (size_t)j * a.ldc : x, ok ? d : 0, sub, hi, lo);
      const double v = fma(-2.0, (double)hi + (double)lo, (double)nbj);
      for (int g = 0; g < kGroups; ++g) {
        const double vg = __shfl_sync(0xffffffffu, v, g * kGroupLanes);
        const int jg = __shfl_sync(0xffffffffu, j, g * kGroupLanes);
        if (!__shfl_sync(0xffffffffu, ok, g * kGroupLanes)) continue;
        if (!(fabs(vg) < 1.0e300)) finite = false;
        if (vg < v1) {
          v2 = v1;
          v1 = vg;
          i1 = jg;
        } else if (vg < v2) {
          v2 = vg;
        }
      }
    }
    const double xn = (double)a.xnorm[pt];
    const double tol = 2.0 * (2.0 * rel * xn * cm + (double)(d + 32) * 0x1p-118) +
                       2.0 * (double)(d + 4) * 0x1p-52 * (xn + cm) * (xn + cm);
    if (i1 >= 0 && finite && (v2 == INFINITY || v2 - v1 > tol)) {
      if (lane == 0) a.labels[pt] = i1;
      continue;
    }
    double best = INFINITY;
    int bidx = -1;
    if (myok) {
      const float* c = a.C + (size_t)myj * a.ldc;
      const double ex = exact_value(1, x, c, d, mynb);
      if (ex < best) {
        best = ex;
        bidx = myj;
      }
    }
    for (int o = 16; o > 0; o >>= 1) {
      const double ob = __shfl_xor_sync(0xffffffffu, best, o);
      const int oi = __shfl_xor_sync(0xffffffffu, bidx, o);
      const bool take = (ob < best) || (ob == best && (unsigned)oi < (unsigned)bidx);
      best = take ? ob : best;
      bidx = take ? oi : bidx;
    }
    if (lane == 0) {
      if (bidx < 0) over[atomicAdd(over_count, 1)] = pt;
      else a.labels[pt] = bidx;
    }
  }
}

// FP64 data: every candidate's exact value, eight lanes (candidates) per point, four points per
// warp: the FP64 pipe takes a warp instruction in the same time whatever its active lanes.
__global__ void resolve_fp64_kernel(ResolveD a) {
  if (grid_enter()) return;
  constexpr int L = 8;
  const long long cnt = min((long long)pinned(a.count), a.max_list);
  const int lane = threadIdx.x & 31, grp = lane / L, sub = lane % L;
  const long long w0 = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const long long nw = ((long long)gridDim.x * blockDim.x) >> 5;
  for (long long s0 = w0 * (32 / L); s0 < cnt; s0 += nw * (32 / L)) {
    const long long slot = s0 + grp;
    const bool live = slot < cnt;
    const int pt = live ? a.list[slot] : 0;
    const int nc = live ? a.cand_cnt[slot] : 0;
    const bool rec = nc > 0 && nc <= kMaxCand;
    double best = INFINITY;
    int bidx = -1;
    if (rec) {
      const double* x = a.X + (size_t)pt * a.ldx;
      for (int q = sub; q < nc; q += L) {
        const int j = a.cand[slot * kMaxCand + q];
        if (j < 0 || j >= a.k) continue;
        const double* c = a.C + (size_t)j * a.c_row;
        double v = 0.0;
        if (a.mode == 0) {
#pragma unroll 8
          for (int t = 0; t < a.d; ++t) {
            const double u = ld(x + t) - ld(c + (size_t)t * a.c_dim);
            v = fma(u, u, v);
          }
        } else {
#pragma unroll 8
          for (int t = 0; t < a.d; ++t) v = fma(ld(x + t), ld(c + (size_t)t * a.c_dim), v);
          v = fma(-2.0, v, a.nb[j]);
        }
        // (a lane's candidates do not come in index order)
        if (v < best || (v == best && bidx >= 0 && j < bidx)) {
          best = v;
          bidx = j;
        }
      }
    }
#pragma unroll
    for (int o = L / 2; o > 0; o >>= 1) {
      const double ob = __shfl_xor_sync(0xffffffffu, best, o);
      const int oi = __shfl_xor_sync(0xffffffffu, bidx, o);
      const bool take = (ob < best) || (ob == best && (unsigned)oi < (unsigned)bidx);
      best = take ? ob : best;
      bidx = take ? oi : bidx;
    }
    if (live && sub == 0) {
      if (bidx < 0) a.over[atomicAdd(a.over_count, 1)] = pt;
      else a.labels[pt] = bidx;
    }
  }
}

// ------------------------------- audit of certified labels -------------------------------
// A rotating sample of rows is checked against the FP64 arg-min over every center, so that a
// failure of a rounding model the certificate relies on (the tensor tiers' accumulation bound,
// the router's separation bound) shows as a counted violation instead of a silently wrong label.
// A violation is a center strictly nearer than the label in FP64 (exact_value, the oracle's
// expression and order); ties are not judged. Distances are first evaluated in FP32, one warp
// per center with the lanes over the dimensions (coalesced rows), each with an interval: any
// summation order of the d non-negative rounded squares stays within (d + 2) 2^-24 relative to
// first order, 2.02x that plus an absolute d 2^-125 for underflow is used. A center whose
// interval lies below the label's is a violation; only overlapping intervals (near ties) are
// decided in FP64, which keeps the narrow FP64 pipe of GB300 out of the scan.
// ws: [0] rows audited, [1] violations, [2] sampling sequence, [3] 1 + the last violating row,
// then per sampled row a violation flag [rows] and the row [rows], and the scan's block ticket in the
// last word.
__device__ __forceinline__ unsigned long long audit_hash(unsigned long long z) {
  z += 0x9E3779B97F4A7C15ull;
  z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
  z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
  return z ^ (z >> 31);
}

// FP32 squared distance of the shared row to center c, lanes over the dimensions (every lane
// returns the warp's sum).
__device__ __forceinline__ float audit_dist32(const float* ax, const float* __restrict__ c, int d,
                                              int lane) {
  float a = 0.0f;
  for (int t = lane; t < d; t += 32) {
    const float u = ax[t] - ld(c + t);
    a = fmaf(u, u, a);
  }
  for (int o = 16; o > 0; o >>= 1) a += __shfl_xor_sync(0xffffffffu, a, o);
  return a;
}

// The same for four consecutive centers j .. j + 3 (clamped to jend - 1), their loads and trees
// interleaved; every center's sum is formed exactly as audit_dist32 forms it.
__device__ __forceinline__ void audit_dist32x4(const float* ax, const float* __restrict__ C,
                                               long long ldc, int j, int jend, int d, int lane,
                                               float out[4]) {
  const float* c[4];
#pragma unroll
  for (int u = 0; u < 4; ++u) {
    c[u] = C + (size_t)min(j + u, jend - 1) * ldc;
    out[u] = 0.0f;
  }
  for (int t = lane; t < d; t += 32) {
    const float xt = ax[t];
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const float v = xt - ld(c[u] + t);
      out[u] = fmaf(v, v, out[u]);
    }
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
#pragma unroll
    for (int u = 0; u < 4; ++u) out[u] += __shfl_xor_sync(0xffffffffu, out[u], o);
  }
}

// The last block of the scan to finish adds up the flags and clears them for the next audit.
__device__ void audit_close(unsigned long long* ws, int rows) {
  __shared__ bool last_sh;
  __shared__ int nviol, naud;
  __shared__ unsigned long long last;
  if (threadIdx.x == 0) {
    __threadfence();
    unsigned int* ticket = reinterpret_cast<unsigned int*>(ws + 4 + 2 * kAuditMaxRows);
    last_sh = atomicAdd(ticket, 1u) == gridDim.x - 1;
    if (last_sh) *ticket = 0;
    __threadfence();
    nviol = 0;
    naud = 0;
    last = 0;
  }
  __syncthreads();
  if (!last_sh) return;
  for (int r = threadIdx.x; r < rows; r += blockDim.x) {
    const unsigned long long row = __ldcg(ws + 4 + rows + r);
    if (row != ~0ull) atomicAdd(&naud, 1);  // not a skipped row
    if (__ldcg(ws + 4 + r)) {
      atomicAdd(&nviol, 1);
      atomicMax(&last, row + 1);
    }
    ws[4 + r] = 0;  // ready for the next audit
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    ws[0] += (unsigned long long)naud;
    ws[1] += (unsigned long long)nviol;
    ws[2] += (unsigned long long)rows;
    if (last) ws[3] = last;
  }
}

__global__ void __launch_bounds__(256)
audit_scan_kernel(const float* X, long long ldx, long long n, int d,
                  const float* C, long long ldc, int k,
                  const int* labels, unsigned long long* ws, int rows, int parts,
                  GroupArgs g, const int* stop) {
  if (grid_enter()) return;
  if (stopped(stop)) return;
  extern __shared__ float ax[];
  __shared__ int viol_sh;
  const int r = blockIdx.x / parts, part = blockIdx.x % parts;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nw = blockDim.x >> 5;
  const unsigned long long seq = *reinterpret_cast<volatile unsigned long long*>(ws + 2);
  const long long row = (long long)(audit_hash(seq + (unsigned long long)r) % (unsigned long long)n);
  // batched problems: the row's problem and its centers; padding rows and rows of stopped
  // problems (their labels belong to the centers before the last update) are not audited
  int cbeg = 0, kk = k;
  if (g.tile_prob) {
    const int prob = g.tile_prob[row >> 7];
    if (row >= g.row_end[prob] || (g.done && g.done[prob])) {  // uniform over the block
      if (threadIdx.x == 0 && part == 0) ws[4 + rows + r] = ~0ull;
      audit_close(ws, rows);
      return;
    }
    cbeg = g.c_off[prob];
    kk = g.k[prob];
  }
  for (int t = threadIdx.x; t < d; t += blockDim.x) ax[t] = X[(size_t)row * ldx + t];
  if (threadIdx.x == 0) viol_sh = 0;
  __syncthreads();
  const float rel = 2.02f * (float)(d + 2) * 5.9604645e-8f;
  const float slack = (float)d * 2.3509887e-38f;  // d 2^-125
  const int lab = labels[row];
  const bool valid = lab >= cbeg && lab < cbeg + kk;
  // the label's interval (every warp evaluates it; an invalid label or one on an unusable
  // center is [inf, inf]: every usable center is nearer)
  float lab_lo = INFINITY, lab_hi = INFINITY;
  if (valid) {
    const float a = audit_dist32(ax, C + (size_t)lab * ldc, d, lane);
    if (a == a) {
      lab_lo = a * (1.0f - rel) - slack;
      lab_hi = a * (1.0f + rel) + slack;
    }
  }
  double dl = -1.0;  // the label's FP64 distance, evaluated when first needed
  const int per = (kk + parts - 1) / parts;
  const int j0 = cbeg + part * per, j1 = min(cbeg + kk, j0 + per);
  bool viol = false;
  for (int jb = j0 + 4 * warp; jb < j1; jb += 4 * nw) {  // four centers per warp step
    float a4[4];
    audit_dist32x4(ax, C, ldc, jb, j1, d, lane, a4);
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const int j = jb + u;
      if (j >= j1 || j == lab) continue;
      const float a = a4[u];
      if (!(a == a)) continue;  // an unusable (NaN) center
      const float lo = a * (1.0f - rel) - slack, hi = a * (1.0f + rel) + slack;
      if (hi < lab_lo) {
        viol = true;
      } else if (lo <= lab_hi && lane == 0) {  // overlapping intervals: decide in FP64
        if (dl < 0.0) {
          dl = valid ? exact_value(0, ax, C + (size_t)lab * ldc, d, 0.0f) : INFINITY;
          if (!(dl == dl)) dl = INFINITY;
        }
        if (exact_value(0, ax, C + (size_t)j * ldc, d, 0.0f) < dl) viol = true;
      }
    }
  }
  if (viol) viol_sh = 1;
  __syncthreads();
  if (threadIdx.x == 0) {
    if (viol_sh) atomicOr(ws + 4 + r, 1ull);
    if (part == 0) ws[4 + rows + r] = (unsigned long long)row;
  }
  audit_close(ws, rows);
}
}  // namespace

cudaError_t launch_gather_flagged(const int* list, const int* count, long long cap,
                                  const void* Xb, const void* Xl, long long row_bytes,
                                  const float* thr, void* XbC, void* XlC, float* thrC, int* over,
                                  int* over_count, const int* stop, cudaStream_t s,
                                  const float* xs, float* xsC) {
  if (inject_fault(kFaultLaunch)) return cudaErrorLaunchOutOfResources;
  if (row_bytes % 16) return cudaErrorInvalidValue;
  launch(gather_flagged_kernel, kmgb::num_sms() * 4, 256, 0, s)(
      list, count, cap, reinterpret_cast<const uint4*>(Xb), reinterpret_cast<const uint4*>(Xl),
      row_bytes / 16, thr, reinterpret_cast<uint4*>(XbC), reinterpret_cast<uint4*>(XlC), thrC, over,
      over_count, stop, xs, xsC);
  count_launches(1);
  return cudaGetLastError();
}

cudaError_t launch_resolve_candidates(const int* list, const int* count, long long max_list,
                                      const int* cand, const int* cand_cnt, const float* X,
                                      long long ldx, const float* C, long long ldc, const float* cn,
                                      int d, int* labels, int* over, int* over_count,
                                      const int* stop, cudaStream_t s, const int* row_map,
                                      const float* hi_in, float* over_hi) {
  if (inject_fault(kFaultLaunch)) return cudaErrorLaunchOutOfResources;
  const bool vec = d % 4 == 0 && ldx % 4 == 0 && ldc % 4 == 0 &&
                   reinterpret_cast<uintptr_t>(X) % 16 == 0 && reinterpret_cast<uintptr_t>(C) % 16 == 0;
  auto kern = vec ? resolve_candidates_kernel<true> : resolve_candidates_kernel<false>;
  launch(kern, kmgb::num_sms() * 8, 256, 0, s)(list, count, max_list, cand, cand_cnt, X, ldx, C, ldc, cn, d,
                                               labels, over, over_count, stop, row_map, hi_in, over_hi,
                                               resolve_tolerances(d));
  count_launches(1);
  return cudaGetLastError();
}

cudaError_t launch_resolve_expansion(const RerankArgs& a, const int* cand, const int* cand_cnt,
                                     int* over, int* over_count, cudaStream_t s) {
  const bool vec = a.d % 4 == 0 && a.ldx % 4 == 0 && a.ldc % 4 == 0 &&
                   reinterpret_cast<uintptr_t>(a.X) % 16 == 0 &&
                   reinterpret_cast<uintptr_t>(a.C) % 16 == 0;
  if (vec)
    launch(resolve_expansion_kernel<true>, kmgb::num_sms() * 8, 256, 0, s)(a, cand, cand_cnt, over,
                                                                       over_count);
  else
    launch(resolve_expansion_kernel<false>, kmgb::num_sms() * 8, 256, 0, s)(a, cand, cand_cnt, over,
                                                                        over_count);
  count_launches(1);
  return cudaGetLastError();
}

cudaError_t launch_resolve_fp64(const ResolveD& a, cudaStream_t s) {
  launch(resolve_fp64_kernel, kmgb::num_sms() * 8, 256, 0, s)(a);
  count_launches(1);
  return cudaGetLastError();
}

static size_t tiled_smem(int d) {
  const int dq = (d + 3) / 4;
  return sizeof(float4) * (size_t)(TP + TC) * ((dq + 1) | 1) + sizeof(float) * TC;
}

bool rerank_tiled_supported(int d) { return tiled_smem(d) <= (size_t)kMaxTileSmem; }

cudaError_t launch_rerank_exact(const RerankArgs& a, const float* hi2, cudaStream_t s) {
  if (inject_fault(kFaultLaunch)) return cudaErrorLaunchOutOfResources;
  if (a.n <= 0 || a.k <= 0) return cudaSuccess;
  const size_t smem = tiled_smem(a.d);
  if (smem > (size_t)kMaxTileSmem || a.mode != 0) return cudaErrorInvalidValue;
  auto kern = rerank_exact_kernel<false>;
  if (smem > kPlainSmem)
    KMGB_CUDA_TRY(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, kMaxTileSmem));
  launch(kern, kmgb::num_sms() * 2, 256, smem, s)(a, hi2, nullptr, nullptr, 0, nullptr, nullptr, nullptr);
  count_launches(1);
  return cudaGetLastError();
}

cudaError_t launch_rerank_band(const RerankArgs& a, const float* hi2, int* cand, int* cand_cnt,
                               long long cand_cap, int* over, int* over_count, float* over_hi,
                               cudaStream_t s) {
  if (inject_fault(kFaultLaunch)) return cudaErrorLaunchOutOfResources;
  if (a.n <= 0 || a.k <= 0) return cudaSuccess;
  const size_t smem = tiled_smem(a.d);
  if (smem > (size_t)kMaxTileSmem || a.mode != 0) return cudaErrorInvalidValue;
  if (smem > kPlainSmem)
    KMGB_CUDA_TRY(cudaFuncSetAttribute(rerank_exact_kernel<true>,
                                       cudaFuncAttributeMaxDynamicSharedMemorySize, kMaxTileSmem));
  launch(rerank_exact_kernel<true>, kmgb::num_sms() * 2, 256, smem, s)(
      a, hi2, cand, cand_cnt, cand_cap, over, over_count, over_hi);
  count_launches(1);
  return cudaGetLastError();
}

cudaError_t launch_rerank_tiled(const RerankArgs& a, int* list2, int* count2, float* hi2,
                                cudaStream_t s) {
  if (inject_fault(kFaultLaunch)) return cudaErrorLaunchOutOfResources;
  if (a.n <= 0 || a.k <= 0) return cudaSuccess;
  const size_t smem = tiled_smem(a.d);
  if (smem > (size_t)kMaxTileSmem || a.mode != 0) return cudaErrorInvalidValue;
  auto kern = rerank_tiled_kernel<0, false>;
  if (smem > kPlainSmem)
    KMGB_CUDA_TRY(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, kMaxTileSmem));
  launch(kern, kmgb::num_sms() * 2, 256, smem, s)(a, list2, count2, hi2);
  count_launches(1);
  return cudaGetLastError();
}

cudaError_t launch_rerank_settle(const RerankArgs& a, cudaStream_t s) {
  if (inject_fault(kFaultLaunch)) return cudaErrorLaunchOutOfResources;
  if (a.n <= 0 || a.k <= 0) return cudaSuccess;
  const size_t smem = tiled_smem(a.d);
  if (smem > (size_t)kMaxTileSmem) return cudaErrorInvalidValue;
  auto kern = a.mode == 0 ? rerank_tiled_kernel<0, true> : rerank_tiled_kernel<1, true>;
  if (smem > kPlainSmem)
    KMGB_CUDA_TRY(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, kMaxTileSmem));
  launch(kern, kmgb::num_sms() * 2, 256, smem, s)(a, nullptr, nullptr, nullptr);
  count_launches(1);
  return cudaGetLastError();
}

cudaError_t launch_rerank_grouped(const RerankArgs& a, const GroupArgs& g, cudaStream_t s,
                                  int* cand, int* cand_cnt, long long cand_cap) {
  if (a.n <= 0 || a.k <= 0) return cudaSuccess;
  if (a.ldc % 4 || (reinterpret_cast<uintptr_t>(a.C) & 15)) return cudaErrorInvalidValue;
  const size_t ds = ((size_t)a.d + 3) / 4 * 4;
  const size_t smem = sizeof(float) * (size_t)RG_WARPS * (RG_VCAP + ds);
  if (smem > (size_t)kMaxTileSmem) return cudaErrorInvalidValue;
  auto kern = a.d <= 16 ? rerank_grouped_kernel<4>
                        : (a.d <= 32 ? rerank_grouped_kernel<8>
                                     : (a.d <= 64 ? rerank_grouped_kernel<16> : rerank_grouped_kernel<32>));
  if (smem > kPlainSmem)
    KMGB_CUDA_TRY(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, kMaxTileSmem));
  launch(kern, kmgb::num_sms() * 4, RG_WARPS * 32, smem, s)(a, g, cand, cand_cnt, cand_cap);
  count_launches(1);
  return cudaGetLastError();
}

cudaError_t launch_rerank(const RerankArgs& a, cudaStream_t s) {
  if (a.n <= 0 || a.k <= 0) return cudaSuccess;
  const int threads = 256;
  const size_t smem = sizeof(float) * (size_t)a.d * (threads / 32);
  if (smem > (size_t)kMaxTileSmem) return cudaErrorInvalidValue;
  if (smem > kPlainSmem) {
    KMGB_CUDA_TRY(cudaFuncSetAttribute(rerank_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       kMaxTileSmem));
  }
  // Persistent grid: the flagged count lives on the device, so no host round trip is needed.
  launch(rerank_kernel, kmgb::num_sms() * 4, threads, smem, s)(a); kmgb::count_launches(1);
  return cudaGetLastError();
}

int audit_parts(int rows) {
  const int p = 8 * kmgb::num_sms() / (rows > 0 ? rows : 1);
  return p < 1 ? 1 : (p > 32 ? 32 : p);
}

cudaError_t launch_audit_labels(const float* X, long long ldx, long long n, int d, const float* C,
                                long long ldc, int k, const int* labels, unsigned long long* ws,
                                int rows, const int* stop, cudaStream_t s, const GroupArgs* grp) {
  if (inject_fault(kFaultLaunch)) return cudaErrorLaunchOutOfResources;
  if (n <= 0 || k <= 0 || rows <= 0) return cudaSuccess;
  if (rows > kAuditMaxRows || (size_t)d * sizeof(float) > 48 * 1024) return cudaErrorInvalidValue;
  const int parts = audit_parts(rows);
  const GroupArgs g = grp ? *grp : GroupArgs{};
  launch(audit_scan_kernel, rows * parts, 256, sizeof(float) * (size_t)d, s)(X, ldx, n, d, C, ldc, k,
                                                                        labels, ws, rows, parts, g,
                                                                        stop);
  count_launches(1);
  return cudaGetLastError();
}

}  // namespace kmgb
