// Plain FP32 fused assignment for sm_103a.
//
// Replaces the reference's register-tiled SGEMM + partial arg-max (main/cuda/ClosestCenters.cu:
// 46-83 with multiply.hcu / reduction.hcu, and _dev_ClosestCentersEndNew :105-123) and the
// cuBLAS + rowTransformMinimum option (kmeans.cpp:918-955). The N x K distance matrix is never
// written:
//   * thread 0 streams 128-point x 32-float tiles of X and 128-center x 32-float tiles of C
//     through a 4-stage shared-memory ring with TMA (128-byte swizzle, mbarrier complete_tx),
//     zero-filling past N, K and D, refilling a stage once all 8 warps released it;
//   * 8 consumer warps accumulate x.c in FP32 FFMA register tiles (8 points x 8 centers per
//     thread, or with the centers' transpose 4 x 16 in packed pairs, the usual case) reading the
//     swizzled tiles bank-conflict free;
//   * per 128-center chunk the epilogue folds d = ||c||^2 - 2 x.c into a running
//     (best, index, second best) per point; the 16 threads sharing a point merge with
//     shuffles, lowest index on ties;
//   * a point is certified when second - best > 2E, E the rigorous rounding bound of the
//     FP32 evaluation; other points are appended to a re-rank list that the exact (FP64)
//     re-rank resolves, so labels equal the FP64 arg-min.
#include <atomic>
#include <cfloat>

#include "common.cuh"
#include "kernels.h"

namespace kmgb {
namespace {

constexpr int BM = 128;        // points per CTA tile
constexpr int BN = 128;        // centers per chunk
constexpr int BKF = 32;        // floats per k-block (128 bytes: one swizzle row)
constexpr int STAGES = 4;
constexpr int NTHREADS = 256;  // 8 warps, all computing; thread 0 also drives TMA
constexpr uint32_t TILE_BYTES = BM * BKF * 4;  // 16 KB (C tile identical)
constexpr uint32_t STAGE_BYTES = 2 * TILE_BYTES;
constexpr size_t SMEM_BYTES = STAGES * STAGE_BYTES + 1024;
constexpr int TSTAGES = 3;     // assign_fp32t_kernel: two CTAs per SM
constexpr size_t TSMEM_BYTES = TSTAGES * STAGE_BYTES + 1024;

__device__ __forceinline__ float bound_e(float xn, float cm, float gamma, int d) {
  // |d~ - (||c||^2 - 2 x.c)| <= u cm^2 + 2 gamma xn cm + u (cm^2 + 2.001 xn cm), plus the FP64
  // reference's own error (d+2) 2^-52 (xn + cm)^2; 1% slack covers FP32 evaluation of E.
  const float u = 5.9604645e-8f;  // 2^-24
  const float xc = xn * cm;
  const float s64 = (float)(d + 2) * 2.220446e-16f * (xn + cm) * (xn + cm);
  const float e = u * cm * cm + 2.0f * gamma * xc + u * (cm * cm + 2.001f * xc) + s64;
  return e * 1.01f + 1e-30f;
}

// The products of four dimensions (16-byte column q of the swizzled tiles) of a thread's 8 points
// and 8 centers.
__device__ __forceinline__ void tile_step(const uint8_t* xs, const uint8_t* cs, int tx, int ty, int q,
                                          float (&acc)[8][8]) {
  float4 cv[8];
#pragma unroll
  for (int j = 0; j < 8; ++j) cv[j] = *reinterpret_cast<const float4*>(cs + swz128(tx + 16 * j, q));
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    const float4 xv = *reinterpret_cast<const float4*>(xs + swz128(ty + 16 * i, q));
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      acc[i][j] = fmaf(xv.x, cv[j].x, acc[i][j]);
      acc[i][j] = fmaf(xv.y, cv[j].y, acc[i][j]);
      acc[i][j] = fmaf(xv.z, cv[j].z, acc[i][j]);
      acc[i][j] = fmaf(xv.w, cv[j].w, acc[i][j]);
    }
  }
}

// One 32-dimension block. TAIL: a row's last block stops at its last 16-byte column (the columns
// past it are zero; at D=324 seven of the last block's eight, 8% of the kernel's work). That second
// loop leaves fewer registers for the first, which is then unrolled by four instead of eight.
template <bool TAIL>
__device__ __forceinline__ void tile_block(const uint8_t* xs, const uint8_t* cs, int tx, int ty,
                                           int dims_left, float (&acc)[8][8]) {
  if (!TAIL) {
#pragma unroll
    for (int q = 0; q < BKF / 4; ++q) tile_step(xs, cs, tx, ty, q, acc);
  } else if (dims_left > BKF - 4) {
#pragma unroll 4
    for (int q = 0; q < BKF / 4; ++q) tile_step(xs, cs, tx, ty, q, acc);
  } else {
#pragma unroll 1
    for (int q = 0; 4 * q < dims_left; ++q) tile_step(xs, cs, tx, ty, q, acc);
  }
}

// Merges the (best, index, second) of the 2 P threads that share P points; the first of them writes the
// label, the bounds and, where the margin does not certify it, the list entry.
template <int P>
__device__ __forceinline__ void settle_tile(const AssignArgs& p, bool compact, long long n_rows,
                                            long long row0, int tx, int ty, float (&b1)[P],
                                            float (&b2)[P], int (&i1)[P]) {
#pragma unroll
  for (int off = 1; off < 2 * P; off <<= 1) {
#pragma unroll
    for (int i = 0; i < P; ++i) {
      const float ob1 = __shfl_xor_sync(0xffffffffu, b1[i], off);
      const float ob2 = __shfl_xor_sync(0xffffffffu, b2[i], off);
      const int oi1 = __shfl_xor_sync(0xffffffffu, i1[i], off);
      const float nb2 = fminf(fminf(b2[i], ob2), fmaxf(b1[i], ob1));
      const bool take = (ob1 < b1[i]) || (ob1 == b1[i] && (unsigned)oi1 < (unsigned)i1[i]);
      b1[i] = take ? ob1 : b1[i];
      i1[i] = take ? oi1 : i1[i];
      b2[i] = nb2;
    }
  }

  if (tx == 0) {
    const float cm = p.certify ? ld(p.cmax) : 0.0f;
#pragma unroll
    for (int i = 0; i < P; ++i) {
      const long long row = row0 + ty + (BM / P) * i;
      if (row < n_rows) {
        const long long pt = compact ? (long long)ld(p.row_map + row) : row;
        p.labels[pt] = i1[i] < 0 ? 0 : i1[i];
        if (p.certify) {
          const float xn = ld(p.xnorm + pt);
          const float e = bound_e(xn, cm, p.gamma, p.d);
          const float margin = b2[i] - b1[i];
          const bool flagged = !(margin > 2.0f * e);
          if (p.ub) {
            // d^2 = ||x||^2 + value, ||x||^2 in [xn^2 (1 - 2^-19), xn^2], every value within e
            const float t1 = __fadd_ru(__fadd_ru(b1[i], e), __fmul_ru(xn, xn));
            const float t2 = __fadd_rd(__fsub_rd(b2[i], e),
                                       __fmul_rd(__fmul_rd(xn, xn), 1.0f - 0x1p-19f));
            p.ub[pt] = flagged ? INFINITY : __fsqrt_ru(fmaxf(t1, 0.0f));
            p.lb[pt] = flagged || !(t2 > 0.0f) ? 0.0f : __fsqrt_rd(t2);
          }
          if (flagged) {
            const int slot = atomicAdd(p.rerank_count, 1);
            p.rerank_list[slot] = (int)pt;
          }
        }
      }
    }
  }
}

template <bool TAIL>
__global__ void __launch_bounds__(NTHREADS, 1)
assign_fp32_kernel(const __grid_constant__ CUtensorMap tmX, const __grid_constant__ CUtensorMap tmC,
                   const __grid_constant__ CUtensorMap tmXc, AssignArgs p) {
  if (grid_enter()) return;
  if (stopped(p.stop)) return;
  // rows present: a device count, or the rows selected by their distance bounds (the compact copy
  // of the listed rows, or all rows when more than its capacity are listed)
  long long n_rows = p.n;
  bool compact = false;
  if (p.n_dev) {
    const long long c = *p.n_dev;
    n_rows = c < p.n ? c : p.n;
  }
  if (p.sel) {
    const int c = *p.sel;
    compact = c <= p.sel_cap;
    if (compact) n_rows = c;
  }
  if ((long long)blockIdx.x * BM >= n_rows) return;  // uniform over the CTA
  extern __shared__ uint8_t smem_raw[];
  // (an offset, not a rounded pointer: the tiles are then known to lie in shared memory)
  uint8_t* smem = smem_raw + ((0u - smem_u32(smem_raw)) & 1023u);
  __shared__ __align__(8) uint64_t full_bar[STAGES];
  __shared__ __align__(8) uint64_t empty_bar[STAGES];
  __shared__ int abort_flag;

  const int tid = threadIdx.x;
  const long long row0 = (long long)blockIdx.x * BM;
  const int nkb = (p.d + BKF - 1) / BKF;
  const int nchunks = (p.k + BN - 1) / BN;
  const int total = nchunks * nkb;

  // Thread 0 doubles as the TMA producer: it fills the ring, then refills each stage as soon
  // as all 8 warps have released it.
  // test hook: steps from p.test_withhold on are never loaded, so the wait for the first of them
  // runs out (every step before it has been loaded and consumed: no copy is left in flight)
  const unsigned long long wait_lim = p.test_wait_cycles ? p.test_wait_cycles : KMGB_WAIT_CYCLES;
  auto issue = [&](int step) {
    if (p.test_withhold > 0 && step >= p.test_withhold) return;
    const int stage = step % STAGES;
    const int chunk = step / nkb, kb = step % nkb;
    const uint32_t dst = smem_u32(smem + stage * STAGE_BYTES);
    const uint32_t bar = smem_u32(&full_bar[stage]);
    mbar_arrive_expect_tx(bar, STAGE_BYTES);
    tma_load_2d(dst, compact ? &tmXc : &tmX, bar, kb * BKF, (int)row0);
    tma_load_2d(dst + TILE_BYTES, &tmC, bar, kb * BKF, chunk * BN);
  };

  if (tid == 0) {
    abort_flag = 0;
    for (int s = 0; s < STAGES; ++s) {
      mbar_init(smem_u32(&full_bar[s]), 1);
      mbar_init(smem_u32(&empty_bar[s]), NTHREADS / 32);
    }
    fence_mbar_init();
    prefetch_tmap(compact ? &tmXc : &tmX);
    prefetch_tmap(&tmC);
  }
  __syncthreads();
  if (tid == 0)
    for (int s = 0; s < STAGES && s < total; ++s) issue(s);

  // ---------------- consumer warps ----------------
  const int lane = tid & 31;
  const int tx = tid & 15;   // center group
  const int ty = tid >> 4;   // point group
  float b1[8], b2[8];
  int i1[8];
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    b1[i] = INFINITY;
    b2[i] = INFINITY;
    i1[i] = -1;
  }

  int s = 0;
  bool alive = true;
  for (int chunk = 0; chunk < nchunks && alive; ++chunk) {
    float acc[8][8];
#pragma unroll
    for (int i = 0; i < 8; ++i)
#pragma unroll
      for (int j = 0; j < 8; ++j) acc[i][j] = 0.0f;

    for (int kb = 0; kb < nkb; ++kb, ++s) {
      const int stage = s % STAGES;
      const uint32_t parity = (s / STAGES) & 1;
      bool ok = mbar_wait(smem_u32(&full_bar[stage]), parity, &abort_flag, p.err,
                          KMGB_DEV_TIMEOUT_FULL, wait_lim);
      ok = __all_sync(0xffffffffu, ok);
      if (!ok) {
        alive = false;
        break;
      }
      const uint8_t* xs = smem + stage * STAGE_BYTES;
      const uint8_t* cs = xs + TILE_BYTES;
      tile_block<TAIL>(xs, cs, tx, ty, p.d - kb * BKF, acc);
      __syncwarp();
      if (lane == 0) mbar_arrive(smem_u32(&empty_bar[stage]));
      if (tid < 32) {  // warp 0: thread 0 refills the stage once every warp released it
        bool ok2 = true;
        if (tid == 0 && s + STAGES < total) {
          ok2 = mbar_wait(smem_u32(&empty_bar[stage]), parity, &abort_flag, p.err,
                          KMGB_DEV_TIMEOUT_EMPTY, wait_lim);
          if (ok2) issue(s + STAGES);
        }
        if (!__all_sync(0xffffffffu, ok2)) {
          alive = false;
          break;
        }
      }
    }
    if (!alive) break;

    // epilogue: fold this chunk into (best, index, second) per point
    float cnv[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      const int c = chunk * BN + tx + 16 * j;
      cnv[j] = (c < p.k) ? ld(p.cn + c) : INFINITY;
    }
#pragma unroll
    for (int i = 0; i < 8; ++i) {
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        const float dv = fmaf(-2.0f, acc[i][j], cnv[j]);
        const float nb2 = fminf(b2[i], fmaxf(b1[i], dv));
        const bool lt = dv < b1[i];
        b1[i] = lt ? dv : b1[i];
        i1[i] = lt ? (chunk * BN + tx + 16 * j) : i1[i];
        b2[i] = nb2;
      }
    }
  }
  if (!alive) return;

  settle_tile(p, compact, n_rows, row0, tx, ty, b1, b2, i1);
}

// ------------------------- transposed centers: packed FP32 products -------------------------
// a += b * c in both halves of a register pair: one instruction for two of the FMAs above.
__device__ __forceinline__ void fma_pair(unsigned long long& a, unsigned long long b,
                                         unsigned long long c) {
  asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(a) : "l"(b), "l"(c));
}
__device__ __forceinline__ unsigned long long twice(float x) {
  unsigned long long r;
  asm("mov.b64 %0, {%1, %1};" : "=l"(r) : "f"(x));
  return r;
}
__device__ __forceinline__ void halves(unsigned long long p, float& lo, float& hi) {
  asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(p));
}

// assign_fp32_kernel over the centers' transpose (tmT: dimension by dimension, 128 centers x 32
// dimensions per stage, unswizzled), so that a dimension's values of neighbouring centers are a register
// pair: a thread's 4 points x 16 centers (4 tx .. 4 tx + 3 of each quarter of the chunk) take 32 packed
// FMAs per dimension instead of 64, and 4 points' values have to be doubled into pairs for them. Every
// (point, center) sum is the same chain in the same order, so the values are bit for bit
// assign_fp32_kernel's. That kernel issues 84% FMAs at 61% of the issue slots (dispatch stalls of
// three-operand FMAs, one CTA of 255 registers a thread per SM) and takes 3.17 ms for 796,160 x 324, K=256;
// this one takes 2.26 ms: 128 registers (64 bytes a thread are spilled), so
// two CTAs hide each other's waits (one CTA: 2.7 ms), and 4 points x 16 centers instead of 8 x 8, which
// doubles half as many values (2.8).
// assign_fp32_kernel stays for centers without a transposed copy (the per-kernel interface).
__global__ void __launch_bounds__(NTHREADS, 2)
assign_fp32t_kernel(const __grid_constant__ CUtensorMap tmX, const __grid_constant__ CUtensorMap tmT,
                    const __grid_constant__ CUtensorMap tmXc, AssignArgs p) {
  if (grid_enter()) return;
  if (stopped(p.stop)) return;
  long long n_rows = p.n;
  bool compact = false;
  if (p.n_dev) {
    const long long c = *p.n_dev;
    n_rows = c < p.n ? c : p.n;
  }
  if (p.sel) {
    const int c = *p.sel;
    compact = c <= p.sel_cap;
    if (compact) n_rows = c;
  }
  if ((long long)blockIdx.x * BM >= n_rows) return;  // uniform over the CTA
  extern __shared__ uint8_t smem_raw[];
  // (an offset, not a rounded pointer: the tiles are then known to lie in shared memory)
  uint8_t* smem = smem_raw + ((0u - smem_u32(smem_raw)) & 1023u);
  __shared__ __align__(8) uint64_t full_bar[TSTAGES];
  __shared__ __align__(8) uint64_t empty_bar[TSTAGES];
  __shared__ int abort_flag;

  const int tid = threadIdx.x;
  const long long row0 = (long long)blockIdx.x * BM;
  const int nkb = (p.d + BKF - 1) / BKF;
  const int nchunks = (p.k + BN - 1) / BN;
  const int total = nchunks * nkb;
  const unsigned long long wait_lim = p.test_wait_cycles ? p.test_wait_cycles : KMGB_WAIT_CYCLES;
  auto issue = [&](int step) {
    if (p.test_withhold > 0 && step >= p.test_withhold) return;
    const int stage = step % TSTAGES;
    const int chunk = step / nkb, kb = step % nkb;
    const uint32_t dst = smem_u32(smem + stage * STAGE_BYTES);
    const uint32_t bar = smem_u32(&full_bar[stage]);
    mbar_arrive_expect_tx(bar, STAGE_BYTES);
    tma_load_2d(dst, compact ? &tmXc : &tmX, bar, kb * BKF, (int)row0);
    tma_load_2d(dst + TILE_BYTES, &tmT, bar, chunk * BN, kb * BKF);
  };
  if (tid == 0) {
    abort_flag = 0;
    for (int s = 0; s < TSTAGES; ++s) {
      mbar_init(smem_u32(&full_bar[s]), 1);
      mbar_init(smem_u32(&empty_bar[s]), NTHREADS / 32);
    }
    fence_mbar_init();
    prefetch_tmap(compact ? &tmXc : &tmX);
    prefetch_tmap(&tmT);
  }
  __syncthreads();
  if (tid == 0)
    for (int s = 0; s < TSTAGES && s < total; ++s) issue(s);

  const int lane = tid & 31;
  constexpr int P = 4;       // points per thread, 64 / P centers
  const int tx = tid & 7;    // center group
  const int ty = tid >> 3;   // point group
  float b1[P], b2[P];
  int i1[P];
#pragma unroll
  for (int i = 0; i < P; ++i) {
    b1[i] = INFINITY;
    b2[i] = INFINITY;
    i1[i] = -1;
  }

  int s = 0;
  bool alive = true;
  for (int chunk = 0; chunk < nchunks && alive; ++chunk) {
    unsigned long long acc[P][8];  // pairs of centers
#pragma unroll
    for (int i = 0; i < P; ++i)
#pragma unroll
      for (int j = 0; j < 8; ++j) acc[i][j] = 0ull;

    for (int kb = 0; kb < nkb; ++kb, ++s) {
      const int stage = s % TSTAGES;
      const uint32_t parity = (s / TSTAGES) & 1;
      bool ok = mbar_wait(smem_u32(&full_bar[stage]), parity, &abort_flag, p.err,
                          KMGB_DEV_TIMEOUT_FULL, wait_lim);
      ok = __all_sync(0xffffffffu, ok);
      if (!ok) {
        alive = false;
        break;
      }
      const uint8_t* xs = smem + stage * STAGE_BYTES;
      const uint8_t* ct = xs + TILE_BYTES + 16 * tx;
      const int nq = min(BKF / 4, (p.d - kb * BKF + 3) / 4);  // the last block stops at its last columns
#pragma unroll 8
      for (int q = 0; q < nq; ++q) {
        float4 xv[P];
#pragma unroll
        for (int i = 0; i < P; ++i)
          xv[i] = *reinterpret_cast<const float4*>(xs + swz128(ty + (BM / P) * i, q));
#pragma unroll
        for (int t = 0; t < 4; ++t) {
          ulonglong2 c[4];
#pragma unroll
          for (int g = 0; g < 4; ++g)
            c[g] = *reinterpret_cast<const ulonglong2*>(ct + (4 * q + t) * (BN * 4) + 128 * g);
#pragma unroll
          for (int i = 0; i < P; ++i) {
            const unsigned long long x =
                twice(t == 0 ? xv[i].x : (t == 1 ? xv[i].y : (t == 2 ? xv[i].z : xv[i].w)));
#pragma unroll
            for (int g = 0; g < 4; ++g) {
              fma_pair(acc[i][2 * g], x, c[g].x);
              fma_pair(acc[i][2 * g + 1], x, c[g].y);
            }
          }
        }
      }
      __syncwarp();
      if (lane == 0) mbar_arrive(smem_u32(&empty_bar[stage]));
      if (tid < 32) {  // warp 0: thread 0 refills the stage once every warp released it
        bool ok2 = true;
        if (tid == 0 && s + TSTAGES < total) {
          ok2 = mbar_wait(smem_u32(&empty_bar[stage]), parity, &abort_flag, p.err,
                          KMGB_DEV_TIMEOUT_EMPTY, wait_lim);
          if (ok2) issue(s + TSTAGES);
        }
        if (!__all_sync(0xffffffffu, ok2)) {
          alive = false;
          break;
        }
      }
    }
    if (!alive) break;

    // epilogue: fold this chunk into (best, index, second) per point
    const int c0 = chunk * BN + 4 * tx;
    // (center j of a thread: 32 (j / 4) + j % 4 past c0)
#pragma unroll
    for (int j = 0; j < 16; ++j) {
      const int c = c0 + (j & 3) + 32 * (j >> 2);
      const float cnv = (c < p.k) ? ld(p.cn + c) : INFINITY;
#pragma unroll
      for (int i = 0; i < P; ++i) {
        float lo, hi;
        halves(acc[i][j >> 1], lo, hi);
        const float dv = fmaf(-2.0f, (j & 1) ? hi : lo, cnv);
        const float nb2 = fminf(b2[i], fmaxf(b1[i], dv));
        const bool lt = dv < b1[i];
        b1[i] = lt ? dv : b1[i];
        i1[i] = lt ? c : i1[i];
        b2[i] = nb2;
      }
    }
  }
  if (!alive) return;
  settle_tile(p, compact, n_rows, row0, tx, ty, b1, b2, i1);
}

// Batched problems of one dimension (GroupArgs): tile t = rows 128t .. 128t+127 belongs to
// problem g.tile_prob[t], whose centers are rows c_off .. c_off + k - 1 of the shared center
// matrix. A persistent grid walks the tiles t = blockIdx.x, += gridDim.x; thread 0 keeps a cursor
// over the flattened (tile, chunk, k-block) steps so the TMA ring runs on across tile boundaries
// (a problem of ~100 centers is one or two chunks: without it every tile would wait for a full
// round trip). Per tile the arithmetic, the fold and the certificate are those of
// assign_fp32_kernel; labels are global center indices; rows past a problem's end (padding to
// its next 128-row boundary) are not written; tiles of stopped problems are skipped.
struct TileCursor {
  long long tile;
  int chunk, kb, cbeg, nchunks;
};

__global__ void __launch_bounds__(NTHREADS, 1)
assign_fp32_grouped_kernel(const __grid_constant__ CUtensorMap tmX,
                           const __grid_constant__ CUtensorMap tmC, AssignArgs p, GroupArgs g,
                           long long ntiles) {
  if (grid_enter()) return;
  extern __shared__ uint8_t smem_raw[];
  // (an offset, not a rounded pointer: the tiles are then known to lie in shared memory)
  uint8_t* smem = smem_raw + ((0u - smem_u32(smem_raw)) & 1023u);
  __shared__ __align__(8) uint64_t full_bar[STAGES];
  __shared__ __align__(8) uint64_t empty_bar[STAGES];
  __shared__ int abort_flag;

  const int tid = threadIdx.x;
  const int nkb = (p.d + BKF - 1) / BKF;
  auto live = [&](long long t) { return !(g.done && g.done[g.tile_prob[t]]); };
  auto first_tile = [&](long long t) {
    while (t < ntiles && !live(t)) t += gridDim.x;
    return t;
  };
  auto open_tile = [&](TileCursor& c, long long t) {
    c.tile = t;
    c.chunk = 0;
    c.kb = 0;
    if (t < ntiles) {
      const int prob = g.tile_prob[t];
      c.cbeg = g.c_off[prob];
      c.nchunks = (g.k[prob] + BN - 1) / BN;
    }
  };
  // producer cursor (thread 0 only)
  TileCursor pc{};
  auto issue_next = [&](int stage) -> bool {
    if (pc.tile >= ntiles) return false;
    const uint32_t dst = smem_u32(smem + stage * STAGE_BYTES);
    const uint32_t bar = smem_u32(&full_bar[stage]);
    mbar_arrive_expect_tx(bar, STAGE_BYTES);
    tma_load_2d(dst, &tmX, bar, pc.kb * BKF, (int)(pc.tile * BM));
    tma_load_2d(dst + TILE_BYTES, &tmC, bar, pc.kb * BKF, pc.cbeg + pc.chunk * BN);
    if (++pc.kb == nkb) {
      pc.kb = 0;
      if (++pc.chunk == pc.nchunks) open_tile(pc, first_tile(pc.tile + gridDim.x));
    }
    return true;
  };

  if (tid == 0) {
    abort_flag = 0;
    for (int s = 0; s < STAGES; ++s) {
      mbar_init(smem_u32(&full_bar[s]), 1);
      mbar_init(smem_u32(&empty_bar[s]), NTHREADS / 32);
    }
    fence_mbar_init();
    prefetch_tmap(&tmX);
    prefetch_tmap(&tmC);
  }
  __syncthreads();
  if (tid == 0) {
    open_tile(pc, first_tile(blockIdx.x));
    for (int s = 0; s < STAGES; ++s)
      if (!issue_next(s)) break;
  }

  const int lane = tid & 31;
  const int tx = tid & 15;
  const int ty = tid >> 4;
  const float cm = p.certify ? ld(p.cmax) : 0.0f;
  long long s = 0;  // steps consumed
  bool alive = true;
  for (long long t = first_tile(blockIdx.x); t < ntiles && alive; t = first_tile(t + gridDim.x)) {
    const int prob = g.tile_prob[t];
    const int cbeg = g.c_off[prob], kp = g.k[prob];
    const long long rend = g.row_end[prob];
    const long long row0 = t * BM;
    const int nchunks = (kp + BN - 1) / BN;
    float b1[8], b2[8];
    int i1[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      b1[i] = INFINITY;
      b2[i] = INFINITY;
      i1[i] = -1;
    }
    for (int chunk = 0; chunk < nchunks && alive; ++chunk) {
      float acc[8][8];
#pragma unroll
      for (int i = 0; i < 8; ++i)
#pragma unroll
        for (int j = 0; j < 8; ++j) acc[i][j] = 0.0f;
      for (int kb = 0; kb < nkb; ++kb, ++s) {
        const int stage = (int)(s % STAGES);
        const uint32_t parity = (uint32_t)((s / STAGES) & 1);
        bool ok = mbar_wait(smem_u32(&full_bar[stage]), parity, &abort_flag, p.err,
                            KMGB_DEV_TIMEOUT_FULL);
        ok = __all_sync(0xffffffffu, ok);
        if (!ok) {
          alive = false;
          break;
        }
        const uint8_t* xs = smem + stage * STAGE_BYTES;
        const uint8_t* cs = xs + TILE_BYTES;
        tile_block<false>(xs, cs, tx, ty, p.d - kb * BKF, acc);
        __syncwarp();
        if (lane == 0) mbar_arrive(smem_u32(&empty_bar[stage]));
        if (tid < 32) {  // warp 0: thread 0 refills the stage once every warp released it
          bool ok2 = true;
          if (tid == 0 && pc.tile < ntiles) {
            ok2 = mbar_wait(smem_u32(&empty_bar[stage]), parity, &abort_flag, p.err,
                            KMGB_DEV_TIMEOUT_EMPTY);
            if (ok2) issue_next(stage);
          }
          if (!__all_sync(0xffffffffu, ok2)) {
            alive = false;
            break;
          }
        }
      }
      if (!alive) break;
      float cnv[8];
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        const int c = chunk * BN + tx + 16 * j;
        cnv[j] = (c < kp) ? ld(p.cn + cbeg + c) : INFINITY;
      }
#pragma unroll
      for (int i = 0; i < 8; ++i) {
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          const float dv = fmaf(-2.0f, acc[i][j], cnv[j]);
          const float nb2 = fminf(b2[i], fmaxf(b1[i], dv));
          const bool lt = dv < b1[i];
          b1[i] = lt ? dv : b1[i];
          i1[i] = lt ? (chunk * BN + tx + 16 * j) : i1[i];
          b2[i] = nb2;
        }
      }
    }
    if (!alive) break;
#pragma unroll
    for (int off = 1; off < 16; off <<= 1) {
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        const float ob1 = __shfl_xor_sync(0xffffffffu, b1[i], off);
        const float ob2 = __shfl_xor_sync(0xffffffffu, b2[i], off);
        const int oi1 = __shfl_xor_sync(0xffffffffu, i1[i], off);
        const float nb2 = fminf(fminf(b2[i], ob2), fmaxf(b1[i], ob1));
        const bool take = (ob1 < b1[i]) || (ob1 == b1[i] && (unsigned)oi1 < (unsigned)i1[i]);
        b1[i] = take ? ob1 : b1[i];
        i1[i] = take ? oi1 : i1[i];
        b2[i] = nb2;
      }
    }
    if (tx == 0) {
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        const long long pt = row0 + ty + 16 * i;
        if (pt < rend) {
          p.labels[pt] = cbeg + (i1[i] < 0 ? 0 : i1[i]);
          if (p.certify) {
            const float e = bound_e(ld(p.xnorm + pt), cm, p.gamma, p.d);
            const float margin = b2[i] - b1[i];
            if (!(margin > 2.0f * e)) {
              const int slot = atomicAdd(p.rerank_count, 1);
              p.rerank_list[slot] = (int)pt;
            }
          }
        }
      }
    }
  }
}

}  // namespace

float assign_fp32_gamma(int d) {
  const double u = 5.9604644775390625e-8;  // 2^-24
  const double g = d * u / (1.0 - d * u);
  return (float)(g * 1.0001);
}

cudaError_t launch_assign_fp32(const float* X, long long ldx, const float* Cop, long long ldc,
                               const AssignArgs& a, cudaStream_t s, const GroupArgs* grp,
                               long long tiles) {
  if (inject_fault(kFaultLaunch)) return cudaErrorLaunchOutOfResources;
  if (a.n <= 0 || a.k <= 0 || a.d <= 0) return cudaSuccess;
  if ((ldx % 4) || (ldc % 4) || (reinterpret_cast<uintptr_t>(X) & 15) ||
      (reinterpret_cast<uintptr_t>(Cop) & 15))
    return cudaErrorInvalidValue;
  CUtensorMap tmX, tmC;
  KMGB_CUDA_TRY(kmgb_make_tmap_2d(&tmX, X, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 4, (uint64_t)a.d,
                                  (uint64_t)a.n, (uint64_t)ldx * 4, BKF, BM));
  KMGB_CUDA_TRY(kmgb_make_tmap_2d(&tmC, Cop, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 4, (uint64_t)a.d,
                                  (uint64_t)a.k, (uint64_t)ldc * 4, BKF, BN));
  static std::atomic<bool> attr_set{false};
  if (!attr_set.load(std::memory_order_acquire)) {
    KMGB_CUDA_TRY(cudaFuncSetAttribute(assign_fp32_kernel<false>,
                                       cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       (int)SMEM_BYTES));
    KMGB_CUDA_TRY(cudaFuncSetAttribute(assign_fp32_kernel<true>,
                                       cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       (int)SMEM_BYTES));
    KMGB_CUDA_TRY(cudaFuncSetAttribute(assign_fp32t_kernel,
                                       cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       (int)TSMEM_BYTES));
    KMGB_CUDA_TRY(cudaFuncSetAttribute(assign_fp32_grouped_kernel,
                                       cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       (int)SMEM_BYTES));
    attr_set.store(true, std::memory_order_release);
  }
  CUtensorMap tmXc = tmX;
  if (a.sel) {
    if (grp || !a.Xc || !a.row_map || a.sel_cap <= 0 || (reinterpret_cast<uintptr_t>(a.Xc) & 15))
      return cudaErrorInvalidValue;
    KMGB_CUDA_TRY(kmgb_make_tmap_2d(&tmXc, a.Xc, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 4, (uint64_t)a.d,
                                    (uint64_t)a.sel_cap, (uint64_t)ldx * 4, BKF, BM));
  }
  if (a.Ct && !grp) {
    CUtensorMap tmT;
    if (a.ldt % 4 || a.ldt < a.k || (reinterpret_cast<uintptr_t>(a.Ct) & 15)) return cudaErrorInvalidValue;
    KMGB_CUDA_TRY(kmgb_make_tmap_2d_swz(&tmT, a.Ct, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 4, (uint64_t)a.k,
                                        (uint64_t)a.d, (uint64_t)a.ldt * 4, BN, BKF,
                                        CU_TENSOR_MAP_SWIZZLE_NONE));
    const long long grid = (a.n + BM - 1) / BM;
    if (grid > 0x7fffffffLL) return cudaErrorInvalidConfiguration;
    launch(assign_fp32t_kernel, (unsigned)grid, NTHREADS, TSMEM_BYTES, s)(tmX, tmT, tmXc, a);
    kmgb::count_launches(1);
    return cudaGetLastError();
  }
  if (grp) {
    if (tiles <= 0) return cudaSuccess;
    if (tiles * BM > a.n) return cudaErrorInvalidConfiguration;
    int dev = 0, sms = 0;
    KMGB_CUDA_TRY(cudaGetDevice(&dev));
    KMGB_CUDA_TRY(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
    const long long grid = tiles < sms ? tiles : sms;
    launch(assign_fp32_grouped_kernel, (unsigned)grid, NTHREADS, SMEM_BYTES, s)(tmX, tmC, a, *grp,
                                                                           tiles);
  } else {
    const long long grid = (a.n + BM - 1) / BM;
    if (grid > 0x7fffffffLL) return cudaErrorInvalidConfiguration;
    const int tail = a.d % BKF;
    if (tail > 0 && tail <= BKF - 4)
      launch(assign_fp32_kernel<true>, (unsigned)grid, NTHREADS, SMEM_BYTES, s)(tmX, tmC, tmXc, a);
    else
      launch(assign_fp32_kernel<false>, (unsigned)grid, NTHREADS, SMEM_BYTES, s)(tmX, tmC, tmXc, a);
  }
  kmgb::count_launches(1);
  return cudaGetLastError();
}

}  // namespace kmgb
