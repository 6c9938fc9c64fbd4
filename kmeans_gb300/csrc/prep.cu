// Per-iteration center preparation and once-per-data-set point preparation.
//
// Replaces the reference's colNormalize (main/cuda/Normalize.cu:33-47, run every iteration from
// kmeans.cpp:1161-1163) and rowNormalize (Normalize.cu:3-31, kmeans.cpp:838-840). Norms are
// accumulated in FP64 and rounded once; an empty-cluster (NaN) center becomes an unusable
// center: zero operand row, +inf norm, so it can never win an arg-min (the reference's
// rowTransformMinimum skips NaN the same way: its val < dataReg is false for NaN,
// RowTransformMinimum.cu:29-31).
#include <cuda_bf16.h>

#include <cuda_fp8.h>

#include <type_traits>

#include "common.cuh"
#include "kernels.h"

namespace kmgb {
namespace {

// Row of the bias matrix (kBiasCols BF16 per center): the start value v split exactly into
// three BF16 numbers, v = hi + mid + lo (v - hi and v - hi - mid are exact in FP32, and what
// is left after two 8-bit pieces of a 24-bit significand fits the third), then zeros.
__device__ __forceinline__ void write_bias_row(__nv_bfloat16* row, float v, int lane) {
  const __nv_bfloat16 hi = __float2bfloat16_rn(v);
  const float r1 = v - __bfloat162float(hi);
  const __nv_bfloat16 mid = __float2bfloat16_rn(r1);
  const __nv_bfloat16 lo = __float2bfloat16_rn(r1 - __bfloat162float(mid));
  if (lane < kBiasCols)
    row[lane] = lane == 0 ? hi : (lane == 1 ? mid : (lane == 2 ? lo : __float2bfloat16_rn(0.0f)));
}

__device__ __forceinline__ void ff_two_sum(float a, float b, float& s, float& e) {
  s = __fadd_rn(a, b);
  const float bp = __fsub_rn(s, a);
  e = __fadd_rn(__fsub_rn(a, __fsub_rn(s, bp)), __fsub_rn(b, bp));
}

__device__ __forceinline__ void ff_square_add(float v, float& hi, float& lo) {
  const float p = __fmul_rn(v, v);
  const float e = __fmaf_rn(v, v, -p);  // v*v - p exactly
  float s, err;
  ff_two_sum(hi, p, s, err);
  hi = s;
  lo = __fadd_rn(lo, __fadd_rn(err, e));
}

// Four squares as a tree, then added: as many operations as one after the other, a shorter chain, and
// smaller errors. ||x||^2's error averages over a cluster's rows into the SSE, with a bias (the low bits of
// squares are not random): relative to the sum, 60,000 rows of Gaussian clusters at D = 16, 32, 64, 128, 300,
// -6.7, -6.9, -6.6, -6.8, -14.4 e-16 one after the other and -5.9, -5.6, -5.7, -5.8, -5.3 e-16 so.
__device__ __forceinline__ void ff_square4_add(float4 v, float& hi, float& lo) {
  const float p0 = __fmul_rn(v.x, v.x), p1 = __fmul_rn(v.y, v.y);
  const float p2 = __fmul_rn(v.z, v.z), p3 = __fmul_rn(v.w, v.w);
  const float e01 = __fadd_rn(__fmaf_rn(v.x, v.x, -p0), __fmaf_rn(v.y, v.y, -p1));
  const float e23 = __fadd_rn(__fmaf_rn(v.z, v.z, -p2), __fmaf_rn(v.w, v.w, -p3));
  float s01, s23, s, t, r01, r23, r, q;
  ff_two_sum(p0, p1, s01, r01);
  ff_two_sum(p2, p3, s23, r23);
  ff_two_sum(s01, s23, s, r);
  const float l = __fadd_rn(__fadd_rn(r01, e01), __fadd_rn(__fadd_rn(r23, e23), r));
  ff_two_sum(hi, s, t, q);
  hi = t;
  lo = __fadd_rn(lo, __fadd_rn(l, q));
}

// Whether float-float (hi, lo), a sum of d squares, lies within its error bound of the middle between two
// FP32 numbers. The bound: (d + 256) 2^-51 of the sum (d / 32 + 8 additions a lane and its tree, each
// 2^-46), taken twice. There the FP64 sum decides, so that every rounded norm is that of the FP64 sum.
__device__ __forceinline__ bool nearly_midway(float hi, float lo, int d) {
  const float e = __fmul_rn(hi, (float)(d + 256) * 0x1p-50f);
  return __fadd_rn(hi, __fadd_rn(lo, e)) != __fadd_rn(hi, __fsub_rn(lo, e));
}

// One warp per center, one pass over its old operand copy and its new values, four dimensions a lane in
// flight. The norm is an error-free float-float sum on the FP32 pipe as a row's (prep_rows_kernel): an
// FP64 chain per lane, its tree and two FP64 square roots in passes of their own took 36.5 us for
// 16,384 x 256 (now 16.9) and 6.6 us for 256 x 128 (4.0).
__global__ void prep_centers_kernel(const float* C, long long ldc, int k, int d,
                                    float* __restrict__ Cop, __nv_bfloat16* __restrict__ Cb,
                                    long long ldcb, float* __restrict__ cn, float* cmax,
                                    const int* stop, float* __restrict__ cinit, int kpad,
                                    __nv_bfloat16* __restrict__ Cl,
                                    __nv_bfloat16* __restrict__ cbias, float* __restrict__ shift,
                                    float* __restrict__ cxn, float shift_pert,
                                    float* __restrict__ Ct, long long ldt) {
  if (grid_enter()) return;
  if (stopped(stop)) return;
  const int warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int lane = threadIdx.x & 31;
  if (warp >= k) {
    if (cinit && warp < kpad && lane == 0) cinit[warp] = -3.0e38f;
    if (cbias && warp < kpad) write_bias_row(cbias + (size_t)warp * kBiasCols, -3.0e38f, lane);
    return;
  }
  const float* c = C + (size_t)warp * ldc;
  float* op = Cop + (size_t)warp * ldc;
  __nv_bfloat16* ob = Cb ? Cb + (size_t)warp * ldcb : nullptr;
  __nv_bfloat16* ol = Cb && Cl ? Cl + (size_t)warp * ldcb : nullptr;
  const int width = ob && ldcb > ldc ? (int)ldcb : (int)ldc;
  float hi = 0.0f, lo = 0.0f;
  float m2 = 0.0f, mx = 0.0f;  // the move since the previous centers
  bool bad = false;
  constexpr int U = 4;
  for (int t0 = lane; t0 < width; t0 += 32 * U) {
    float v[U], o[U];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int t = t0 + 32 * u;
      v[u] = t < d ? c[t] : 0.0f;
      o[u] = shift && t < d ? op[t] : 0.0f;
    }
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int t = t0 + 32 * u;
      bad |= !isfinite(v[u]);
      ff_square_add(v[u], hi, lo);
      if (shift) {
        const float df = fabsf(v[u] - o[u]);
        m2 = fmaf(df, df, m2);
        mx = fmaxf(mx, df);
      }
      if (t < (int)ldc) op[t] = v[u];
      if (Ct && t < d) Ct[(size_t)t * ldt + warp] = v[u];
      if (ob && t < (int)ldcb) {
        const __nv_bfloat16 h = __float2bfloat16_rn(v[u]);
        ob[t] = h;
        if (ol) ol[t] = __float2bfloat16_rn(v[u] - __bfloat162float(h));
      }
    }
  }
  bad = __any_sync(0xffffffffu, bad);
  if (bad) {  // unusable: zero operands
    for (int t = lane; t < width; t += 32) {
      if (t < (int)ldc) op[t] = 0.0f;
      if (Ct && t < d) Ct[(size_t)t * ldt + warp] = 0.0f;
      if (ob && t < (int)ldcb) {
        ob[t] = __float2bfloat16_rn(0.0f);
        if (ol) ol[t] = __float2bfloat16_rn(0.0f);
      }
    }
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    const float oh = __shfl_xor_sync(0xffffffffu, hi, o);
    const float olo = __shfl_xor_sync(0xffffffffu, lo, o);
    float s1, err;
    ff_two_sum(hi, oh, s1, err);
    hi = s1;
    lo = __fadd_rn(lo, __fadd_rn(olo, err));
    if (shift) {
      m2 += __shfl_xor_sync(0xffffffffu, m2, o);
      mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
    }
  }
  // the squared norm, and an upper bound of the norm. The lanes' lo parts may differ in their last bits
  // (the butterfly adds them in another order on either side): one lane's serve all, since the lanes
  // write parts of one number below
  lo = __shfl_sync(0xffffffffu, lo, 0);
  float nn = __fadd_rn(hi, lo);
  float nrm = __fsqrt_ru(__fmul_ru(__fadd_ru(hi, fabsf(lo)), 1.0f + 0x1p-22f));
  // squares out of FP32's normal range, or a norm halfway between two FP32 numbers (uniform)
  if (!bad && (!(hi < 1.0e37f && hi >= 1.0e-24f) || nearly_midway(hi, lo, d))) {
    double s = 0.0;
    for (int t = lane; t < d; t += 32) s = fma((double)c[t], (double)c[t], s);
    for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    nn = __double2float_rn(s);
    nrm = __double2float_ru(sqrt(s) * (1.0 + 1e-12));
  }
  if (cbias) write_bias_row(cbias + (size_t)warp * kBiasCols, bad ? -3.0e38f : -0.5f * nn, lane);
  if (lane != 0) return;
  if (shift) {
    // FP32 sum of squared differences, widened by more than its roundings; where squares leave the
    // normal range, sqrt(d) times the largest difference
    const bool was_bad = !(cn[warp] < INFINITY);
    const float slack = 1.0f + (float)(d + 16) * 2.4e-7f;
    const float mv = (mx == 0.0f || (m2 > 1e-28f && m2 < 1e37f))
                         ? __fsqrt_ru(__fmul_ru(m2, slack))
                         : __fmul_ru(__fmul_ru(mx, 1.000001f), __fsqrt_ru((float)d));
    // FP64 centers: each end of the move is a rounding away from its center
    const float pt = shift_pert > 0.0f ? __fmul_ru(shift_pert, __fadd_ru(nrm, mv)) : 0.0f;
    shift[warp] = bad && was_bad ? -1.0f : (bad || was_bad ? INFINITY : __fadd_ru(mv, pt));
  }
  if (bad) {
    cn[warp] = INFINITY;
    if (cxn) cxn[warp] = 0.0f;
    if (cinit) cinit[warp] = -3.0e38f;
  } else {
    cn[warp] = nn;
    if (cinit) cinit[warp] = -0.5f * nn;
    atomicMax(reinterpret_cast<int*>(cmax), __float_as_int(nrm));
    if (cxn) cxn[warp] = nrm;
  }
}

// Everything an iteration needs of a row, from one read of it: qn = ||x||^2 (FP64), xn = FP32 upper
// bound of ||x||, the BF16 value plane and its residual plane bf16(x - bf16(x)) (each nullable).
// GB300's FP64 pipe is narrow, so the norm runs on the FP32 pipe as an error-free float-float value:
// exact squares (p + e by FMA), TwoSum accumulation per lane, a float-float tree over the lanes, and
// a single FP64 addition per row; it is within (d/32 + 8) 2^-46 of ||x||^2 relative, and xn adds
// 2^-20 before its upward-rounded square root. Rows whose squares leave the FP32 range are summed
// in FP64 instead. inexact (nullable): set to 1 when some value is not a BF16 number (v != bf16(v);
// NaN included), i.e. when the residual plane carries information.
//
// Bound by HBM: 4 bytes read and 4 written per element. L lanes share a row, each with 16 bytes of
// it at a time (L = 32 from 68 dimensions on, fewer below, so that a warp's lanes are all busy and
// its loads contiguous), and a warp takes two row groups at a time. One pass per kind of output with
// a warp and 4 bytes a lane per row took 153 + 69 us for 898,790 x 128 (norms, one plane pair);
// the tree and the row's results one row at a time, and FP64 conversions that the compiler ran with qn
// null too, 52 us for 224,698 x 128 (now 40).
// T = double: the FP32 roundings of FP64 rows (row stride ldx doubles, read element by element
// unless rows are 16-byte aligned).
template <typename T>
__device__ __forceinline__ float4 load_row4(const T* __restrict__ x, int c, int d, bool vec) {
  float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
  if (sizeof(T) == 4) {
    if (vec && c + 4 <= d) return ld(reinterpret_cast<const float4*>(x + c));
  } else if (vec && c + 4 <= d) {
    const double2 a = ld(reinterpret_cast<const double2*>(x + c));
    const double2 b = ld(reinterpret_cast<const double2*>(x + c + 2));
    return make_float4(__double2float_rn(a.x), __double2float_rn(a.y), __double2float_rn(b.x),
                       __double2float_rn(b.y));
  }
  if (c < d) v.x = (float)ld(x + c);
  if (c + 1 < d) v.y = (float)ld(x + c + 1);
  if (c + 2 < d) v.z = (float)ld(x + c + 2);
  if (c + 3 < d) v.w = (float)ld(x + c + 3);
  return v;
}

__device__ __forceinline__ uint2 bf16x4(float4 v) {
  const __nv_bfloat162 a = __floats2bfloat162_rn(v.x, v.y), b = __floats2bfloat162_rn(v.z, v.w);
  return make_uint2(*reinterpret_cast<const uint32_t*>(&a), *reinterpret_cast<const uint32_t*>(&b));
}
// the values of the four BF16 numbers
__device__ __forceinline__ float4 widen4(uint2 b) {
  return make_float4(__uint_as_float(b.x << 16), __uint_as_float(b.x & 0xFFFF0000u),
                     __uint_as_float(b.y << 16), __uint_as_float(b.y & 0xFFFF0000u));
}

//
// IDX 1: the rows of a device list (RowList): output row i is row list[i]; entries past the capacity
// go to over. IDX 2: a mini-batch window (RowWindow), whose rows are copied on the way (gathering the
// rows, their norms and their planes were three launches: 32 + 6 + 19 us for 89,879 x 128).
template <typename T, int L, int IDX>
__global__ void __launch_bounds__(256)
prep_rows_kernel(const T* X, long long ldx, long long n, int d, bool vec,
                 double* __restrict__ qn, float* __restrict__ xn, uint2* __restrict__ Xb,
                 uint2* __restrict__ Xl, int ldb, int* inexact, float* __restrict__ nf, RowList rl,
                 RowWindow rw, const int* stop) {
  if (grid_enter()) return;
  if (stopped(stop)) return;
  if (IDX == 1) {
    const long long total = pinned(rl.count);
    const long long cap = n;
    n = total < cap ? total : cap;
    for (long long i = cap + (long long)blockIdx.x * blockDim.x + threadIdx.x; i < total;
         i += (long long)gridDim.x * blockDim.x)
      rl.over[atomicAdd(rl.over_count, 1)] = rl.list[i];
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n;
         i += (long long)gridDim.x * blockDim.x) {
      const float fl = rl.thr[rl.list[i]];  // without a finite floor: no candidates (gather_flagged_kernel)
      rl.thr_out[i] = fl > -3.0e38f ? fl : __int_as_float(0x7fc00000);
    }
  }
  long long start = 0;
  if (IDX == 2) start = (((long long)*rw.base + *rw.done) * n) % rw.m;
  auto source = [&](long long r) -> long long {
    if (IDX == 1) return ld(rl.list + r);
    if (IDX == 2) {
      const long long pos = start + r;
      return ld(rw.perm + (pos >= rw.m ? pos - rw.m : pos));
    }
    return r;
  };
  constexpr int G = 32 / L;  // rows per warp and step
  constexpr int U = 2;       // steps in flight
  const int lane = threadIdx.x & 31, grp = lane / L, sub = lane % L;
  const long long w0 = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const long long nw = ((long long)gridDim.x * blockDim.x) >> 5;
  const int ldb4 = ldb / 4;
  int width = Xb ? ldb : d;  // planes are written with their zero padding
  if (IDX == 2 && rw.ld_out > width) width = (int)rw.ld_out;
  const bool norms = qn || xn || nf;
  bool off = false;
  for (long long r0 = w0 * G * U; r0 < n; r0 += nw * G * U) {
    float hi[U], lo[U];
#pragma unroll
    for (int u = 0; u < U; ++u) hi[u] = lo[u] = 0.0f;
    for (int c = 4 * sub; c < width; c += 4 * L) {
      float4 v[U];
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const long long r = r0 + u * G + grp;
        v[u] = r < n ? load_row4(X + (size_t)source(r) * ldx, c, d, vec) : make_float4(0.f, 0.f, 0.f, 0.f);
      }
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const long long r = r0 + u * G + grp;
        if (norms) ff_square4_add(v[u], hi[u], lo[u]);
        if (IDX == 2 && r < n && c < rw.ld_out)
          *reinterpret_cast<float4*>(rw.X_out + (size_t)r * rw.ld_out + c) = v[u];
        if (Xb && r < n && c < ldb) {
          const uint2 h = bf16x4(v[u]);
          Xb[(size_t)r * ldb4 + c / 4] = h;
          if (Xl || inexact) {
            const float4 hv = widen4(h);
            if (inexact) off |= !(v[u].x == hv.x && v[u].y == hv.y && v[u].z == hv.z && v[u].w == hv.w);
            if (Xl)
              Xl[(size_t)r * ldb4 + c / 4] = bf16x4(make_float4(v[u].x - hv.x, v[u].y - hv.y,
                                                                v[u].z - hv.z, v[u].w - hv.w));
          }
        }
      }
    }
    if (!norms) continue;
    // the two rows' trees: the first step leaves the first row's to the lower half of the lanes and the
    // second's to the upper half (each adding its pair as lane 0 would), the others run on one value
    static_assert(U == 2, "a row per half");
    constexpr int H = L / 2;
    const bool up = sub >= H;
    const long long r = r0 + (up ? G : 0) + grp;
    float h1, l1;
    {
      const float oh = __shfl_xor_sync(0xffffffffu, up ? hi[0] : hi[1], H);
      const float ol = __shfl_xor_sync(0xffffffffu, up ? lo[0] : lo[1], H);
      const float mh = up ? hi[1] : hi[0], ml = up ? lo[1] : lo[0];
      float err;
      ff_two_sum(up ? oh : mh, up ? mh : oh, h1, err);
      l1 = __fadd_rn(up ? ol : ml, __fadd_rn(up ? ml : ol, err));
    }
#pragma unroll
    for (int o = H / 2; o > 0; o >>= 1) {
      const float oh = __shfl_xor_sync(0xffffffffu, h1, o);
      const float ol = __shfl_xor_sync(0xffffffffu, l1, o);
      float s1, err;
      ff_two_sum(h1, oh, s1, err);
      h1 = s1;
      l1 = __fadd_rn(l1, __fadd_rn(ol, err));
    }
    // overflow (or NaN input): FP64 sum; for the rounded norm also where squares near the
    // subnormals lose their low parts, and where its rounding could differ from the FP64 sum's
    const bool wide = !(fabsf(h1) < 1.0e37f) || (nf && (h1 < 1.0e-24f || nearly_midway(h1, l1, d)));
    if (__any_sync(0xffffffffu, wide)) {
#pragma unroll 1
      for (int u = 0; u < U; ++u) {
        const long long ru = r0 + u * G + grp;
        double sd = 0.0;
        if (ru < n)
          for (int t = sub; t < d; t += L) {
            const double x = (double)(float)ld(X + (size_t)source(ru) * ldx + t);
            sd = fma(x, x, sd);
          }
        for (int o = L / 2; o > 0; o >>= 1) sd += __shfl_xor_sync(0xffffffffu, sd, o);
        if (wide && sub == u * H && ru < n) {
          if (qn) qn[ru] = sd;
          if (nf) nf[ru] = __double2float_rn(sd);
          if (xn) xn[ru] = __double2float_ru(sqrt(sd) * (1.0 + 1e-12));
        }
      }
    }
    if (!wide && (sub == 0 || sub == H) && r < n) {
      if (qn) {
        asm volatile("" : "+f"(h1));  // (keeps the FP64 conversions from running where qn is null)
        qn[r] = (double)h1 + (double)l1;
      }
      if (nf) nf[r] = __fadd_rn(h1, l1);
      if (xn) xn[r] = __fsqrt_ru(__fmul_ru(__fadd_ru(h1, fabsf(l1)), 1.0f + 0x1p-20f));
    }
  }
  if (inexact && __any_sync(0xffffffffu, off) && lane == 0) atomicExch(inexact, 1);
}

// Centers of the expansion form (per-kernel ABI: B is d x k, centers are columns, with the caller's
// norms nb): one warp per center writes the row-major FP32 copy Bt, nbx = the norm or +inf where the
// center can never win (a NaN anywhere, a norm of +inf), the BF16 planes and the start values -nb/2
// (nullable), and raises *cmax >= max(||c||, sqrt|nb|). A center whose value no bound covers
// (infinite elements, a norm of -inf, magnitudes beyond 1e18) raises it to 3e38: every row then
// misses its certificate and is settled exactly.
template <typename T>
__global__ void prep_expansion_kernel(const T* B, int d, int k, const T* nb,
                                      float* __restrict__ Bt, long long ld, float* __restrict__ nbx,
                                      __nv_bfloat16* __restrict__ Cb, __nv_bfloat16* __restrict__ Cl,
                                      long long ldb, float* __restrict__ cinit,
                                      __nv_bfloat16* __restrict__ cbias, int kpad, float* cmax) {
  if (grid_enter()) return;
  const int j = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int lane = threadIdx.x & 31;
  if (j >= kpad) return;
  float start = -3.0e38f;
  if (j < k) {
    double s = 0.0;
    bool nan = false, wide = false;
    for (int t = lane; t < d; t += 32) {
      const T v = B[(size_t)t * k + j];
      nan |= v != v;
      wide |= !(fabs((double)v) < 1e18);
      s = fma((double)v, (double)v, s);
    }
    for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    const T n = nb[j];
    nan = __any_sync(0xffffffffu, nan) || n != n;
    wide = __any_sync(0xffffffffu, wide);
    const bool never = nan || (!wide && n > T(0) && !(n < (T)INFINITY));
    const bool force = !never && (wide || !(fabs((double)n) < 1e36));
    const bool zero = never || force;
    for (int t = lane; t < (int)ld; t += 32)
      Bt[(size_t)j * ld + t] = (never || t >= d) ? 0.0f : (float)B[(size_t)t * k + j];
    if (Cb)
      for (int t = lane; t < (int)ldb; t += 32) {
        const float v = (zero || t >= d) ? 0.0f : (float)B[(size_t)t * k + j];
        const __nv_bfloat16 hi = __float2bfloat16_rn(v);
        Cb[(size_t)j * ldb + t] = hi;
        Cl[(size_t)j * ldb + t] = __float2bfloat16_rn(v - __bfloat162float(hi));
      }
    if (!zero) start = -0.5f * (float)n;
    if (lane == 0) {
      nbx[j] = never ? INFINITY : (float)n;
      if (!never) {
        const float up = force ? 3.0e38f
                               : __double2float_ru(sqrt(fmax(s, fabs((double)n))) * (1.0 + 1e-12));
        atomicMax(reinterpret_cast<int*>(cmax), __float_as_int(up));
      }
    }
  }
  if (cinit && lane == 0) cinit[j] = start;
  if (cbias) write_bias_row(cbias + (size_t)j * kBiasCols, start, lane);
}

// FP8 E4M3 operands with power-of-two scales: x = s * x8 + error, s = 2^(e - 8) where the scaled
// quantity (a row's largest |x_i|, or for the centers the largest ||c||) is below 2^e, so every
// scaled value is below 2^8 = 256 < 448 (the largest E4M3 number: no saturation) and the division
// by s is exact; the conversion rounds to nearest even, each element within 2^-4 relative of its
// value when normal and within s 2^-10 when it falls among the subnormals.
__device__ __forceinline__ float pow2_scale_for(float mx) {
  if (!(mx > 0.0f) || !(mx < INFINITY)) return 1.0f;
  int e;
  frexpf(mx, &e);  // mx = f 2^e, f in [0.5, 1)
  return ldexpf(1.0f, e - 8);
}

// One warp per row: the row's scale (sx[row]) and its E4M3 copy, zero padded to ld8 bytes.
__global__ void to_fp8_kernel(const float* X, long long ldx, long long n, int d,
                              uint8_t* __restrict__ X8, long long ld8, float* __restrict__ sx,
                              const int* stop) {
  if (grid_enter()) return;
  if (stopped(stop)) return;
  const int lane = threadIdx.x & 31;
  for (long long r = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5; r < n;
       r += ((long long)gridDim.x * blockDim.x) >> 5) {
    const float* x = X + (size_t)r * ldx;
    float mx = 0.0f;
    for (int t = lane; t < d; t += 32) mx = fmaxf(mx, fabsf(x[t]));
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
    const float sc = pow2_scale_for(mx);
    const float inv = 1.0f / sc;  // a power of two: exact
    for (long long t = lane; t < ld8; t += 32)
      X8[(size_t)r * ld8 + t] =
          t < d ? (uint8_t)__nv_cvt_float_to_fp8(x[t] * inv, __NV_SATFINITE, __NV_E4M3) : 0;
    if (lane == 0) sx[r] = sc;
  }
}

// The centers' E4M3 copy with one scale for all of them, from the operand copy (unusable centers
// are zero rows) and the bound of the largest center norm: cscale = 2^(e - 8), cmax < 2^e.
__global__ void centers_fp8_kernel(const float* Cop, long long ldc, int k, int d,
                                   const float* cmax, uint8_t* __restrict__ C8,
                                   long long ld8, float* __restrict__ cscale, const int* stop) {
  if (grid_enter()) return;
  if (stopped(stop)) return;
  const float sc = pow2_scale_for(*cmax);
  const float inv = 1.0f / sc;
  if (blockIdx.x == 0 && threadIdx.x == 0) *cscale = sc;
  const long long total = (long long)k * ld8;
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < total;
       i += (long long)gridDim.x * blockDim.x) {
    const long long c = i / ld8, t = i % ld8;
    C8[i] = t < d ? (uint8_t)__nv_cvt_float_to_fp8(Cop[(size_t)c * ldc + t] * inv,
                                                     __NV_SATFINITE, __NV_E4M3)
                  : 0;
  }
}

}  // namespace

cudaError_t launch_to_fp8(const float* X, long long ldx, long long n, int d, void* X8,
                          long long ld8, float* sx, cudaStream_t s, const int* stop) {
  if (inject_fault(kFaultLaunch)) return cudaErrorLaunchOutOfResources;
  if (n <= 0) return cudaSuccess;
  if (ld8 % 16 || ld8 < d) return cudaErrorInvalidValue;
  launch(to_fp8_kernel, kmgb::num_sms() * 16, 256, 0, s)(X, ldx, n, d, static_cast<uint8_t*>(X8), ld8,
                                                     sx, stop);
  kmgb::count_launches(1);
  return cudaGetLastError();
}

cudaError_t launch_centers_fp8(const float* Cop, long long ldc, int k, int d, const float* cmax,
                               void* C8, long long ld8, float* cscale, cudaStream_t s,
                               const int* stop) {
  if (k <= 0) return cudaSuccess;
  if (ld8 % 16 || ld8 < d) return cudaErrorInvalidValue;
  launch(centers_fp8_kernel, kmgb::num_sms() * 4, 256, 0, s)(Cop, ldc, k, d, cmax,
                                                         static_cast<uint8_t*>(C8), ld8, cscale,
                                                         stop);
  kmgb::count_launches(1);
  return cudaGetLastError();
}

cudaError_t launch_prep_centers(const float* C, long long ldc, int k, int d, float* Cop, void* Cb,
                                long long ldcb, float* cn, float* cmax, cudaStream_t s,
                                const int* stop, float* cinit, void* Cl, void* cbias,
                                float* shift, float* cxn, float shift_pert, float* Ct,
                                long long ldt) {
  if (inject_fault(kFaultLaunch)) return cudaErrorLaunchOutOfResources;
  if (k <= 0) return cudaSuccess;
  const int threads = 256;
  const int kpad = (k + kCenterPad - 1) / kCenterPad * kCenterPad;
  const int blocks = (int)(((long long)(cinit || cbias ? kpad : k) * 32 + threads - 1) / threads);
  launch(prep_centers_kernel, blocks, threads, 0, s)(C, ldc, k, d, Cop,
                                                 reinterpret_cast<__nv_bfloat16*>(Cb), ldcb, cn,
                                                 cmax, stop, cinit, kpad,
                                                 reinterpret_cast<__nv_bfloat16*>(Cl),
                                                 reinterpret_cast<__nv_bfloat16*>(cbias), shift,
                                                 cxn, shift_pert, Ct, ldt);
  kmgb::count_launches(1);
  return cudaGetLastError();
}

template <typename T>
static cudaError_t prep_rows(const T* X, long long ldx, long long n, int d, double* qn, float* xn,
                             void* Xb, void* Xl, long long ldb, int* inexact, float* nf,
                             cudaStream_t s, const int* stop, const RowList* rl,
                             const RowWindow* rw = nullptr) {
  if (inject_fault(kFaultLaunch)) return cudaErrorLaunchOutOfResources;
  if (n <= 0) return cudaSuccess;
  if (Xb && (ldb % 8 || ldb < d)) return cudaErrorInvalidValue;
  const bool vec = (ldx * sizeof(T)) % 16 == 0 && reinterpret_cast<uintptr_t>(X) % 16 == 0;
  const int lanes = d <= 16 ? 4 : (d <= 32 ? 8 : (d <= 64 ? 16 : 32));
  const long long steps = (n + 2 * (32 / lanes) - 1) / (2 * (32 / lanes));  // warps' worth of rows
  const long long most = kmgb::num_sms() * 64LL;
  const unsigned blocks = (unsigned)((steps < most ? steps : most) + 7) / 8;
  uint2* b = static_cast<uint2*>(Xb);
  uint2* l = static_cast<uint2*>(Xl);
  auto go = [&](auto tag) {
    if (rl)
      launch(prep_rows_kernel<T, decltype(tag)::value, 1>, blocks, 256, 0, s)(
          X, ldx, n, d, vec, qn, xn, b, l, (int)ldb, inexact, nullptr, *rl, RowWindow{}, stop);
    else if (rw)
      launch(prep_rows_kernel<T, decltype(tag)::value, 2>, blocks, 256, 0, s)(
          X, ldx, n, d, vec, qn, xn, b, l, (int)ldb, inexact, nullptr, RowList{}, *rw, stop);
    else
      launch(prep_rows_kernel<T, decltype(tag)::value, 0>, blocks, 256, 0, s)(
          X, ldx, n, d, vec, qn, xn, b, l, (int)ldb, inexact, nf, RowList{}, RowWindow{}, stop);
  };
  if (lanes == 4) go(std::integral_constant<int, 4>{});
  else if (lanes == 8) go(std::integral_constant<int, 8>{});
  else if (lanes == 16) go(std::integral_constant<int, 16>{});
  else go(std::integral_constant<int, 32>{});
  kmgb::count_launches(1);
  return cudaGetLastError();
}
template <typename T>
cudaError_t launch_prep_rows(const T* X, long long ldx, long long n, int d, double* qn, float* xn,
                             void* Xb, void* Xl, long long ldb, int* inexact, cudaStream_t s,
                             const int* stop, const RowList* rl) {
  return prep_rows<T>(X, ldx, n, d, qn, xn, Xb, Xl, ldb, inexact, nullptr, s, stop, rl);
}

cudaError_t launch_prep_window(const float* X, long long ldx, long long n, int d, double* qn, float* xn,
                               void* Xb, void* Xl, long long ldb, const RowWindow& rw, cudaStream_t s,
                               const int* stop) {
  if (rw.ld_out % 4 || rw.ld_out < d || (reinterpret_cast<uintptr_t>(rw.X_out) & 15) || n > rw.m)
    return cudaErrorInvalidValue;
  return prep_rows<float>(X, ldx, n, d, qn, xn, Xb, Xl, ldb, nullptr, nullptr, s, stop, nullptr, &rw);
}

cudaError_t launch_row_norms(const float* X, long long ldx, long long n, int d, float* out,
                             cudaStream_t s) {
  return prep_rows<float>(X, ldx, n, d, nullptr, nullptr, nullptr, nullptr, 0, nullptr, out, s, nullptr,
                          nullptr);
}

template cudaError_t launch_prep_rows<float>(const float*, long long, long long, int, double*, float*,
                                             void*, void*, long long, int*, cudaStream_t, const int*,
                                             const RowList*);
template cudaError_t launch_prep_rows<double>(const double*, long long, long long, int, double*,
                                              float*, void*, void*, long long, int*, cudaStream_t,
                                              const int*, const RowList*);

template <typename T>
cudaError_t launch_prep_expansion(const T* B, int d, int k, const T* nb, float* Bt, long long ld,
                                  float* nbx, void* Cb, void* Cl, long long ldb, float* cinit,
                                  void* cbias, float* cmax, cudaStream_t s) {
  const int kpad = cinit ? (k + kCenterPad - 1) / kCenterPad * kCenterPad : k;
  launch(prep_expansion_kernel<T>, (unsigned)(((long long)kpad * 32 + 255) / 256), 256, 0, s)(
      B, d, k, nb, Bt, ld, nbx, static_cast<__nv_bfloat16*>(Cb), static_cast<__nv_bfloat16*>(Cl), ldb,
      cinit, static_cast<__nv_bfloat16*>(cbias), kpad, cmax);
  kmgb::count_launches(1);
  return cudaGetLastError();
}
template cudaError_t launch_prep_expansion<float>(const float*, int, int, const float*, float*,
                                                  long long, float*, void*, void*, long long, float*,
                                                  void*, float*, cudaStream_t);
template cudaError_t launch_prep_expansion<double>(const double*, int, int, const double*, float*,
                                                   long long, float*, void*, void*, long long, float*,
                                                   void*, float*, cudaStream_t);

}  // namespace kmgb
