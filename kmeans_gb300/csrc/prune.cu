// Distance bounds kept from one iteration of a run to the next (Hamerly, "Making k-means even
// faster", SDM 2010): rows whose label is proved without looking at the centers again.
//
// The assignment leaves, for every row whose label its certificate proves, an upper bound ub of the
// distance to the label's center and a lower bound lb of the distance to every other usable center
// (directed rounding, the tier's error bound included). When the centers move, ub grows by the
// move of the row's own center and lb shrinks by the largest move of the others; half the distance
// from a center to its nearest other center (from one scan of the centers against themselves) is a
// second threshold. While ub stays below the larger of the two, every other center is strictly
// farther, so the label is still the FP64 arg-min and the row is not scanned; the other rows are
// copied to a compact matrix and scanned as ever. A center none of whose rows changed keeps its
// sums, its place and its SSE terms: the update is deterministic, so they would come out the same. The
// reference scans every row in every iteration (kmeans.cpp:910-1014). Nothing survives a run: its first
// iteration scans every row.
//
// prune_filter_kernel is bound by HBM: 12 bytes read and 8 written per row.
#include <cstdlib>
#include <cstring>

#include "common.cuh"
#include "kernels.h"

namespace kmgb {
namespace {

constexpr int PF_THREADS = 256;
constexpr int PF_ROWS = 4 * PF_THREADS;  // rows per block step, four consecutive ones per thread

// The two largest moves and the center of the largest (unusable centers, -1, never count); starts
// the list of rows to scan: empty when the rows are tested, else past every capacity (and every
// center's members count as changed). One block.
// State (flags[7]): bit 0, this iteration scans every row untested; bit 1, lab_old is not that of the last
// update; bits 8 up, iterations yet to go untested; bits 16 up, how many the last failed test asked for.
__global__ void __launch_bounds__(1024)
prune_top_kernel(PruneState ps, const int* stop) {
  if (grid_enter()) return;
  if (stopped(stop)) return;
  __shared__ float s1[32], s2[32];
  __shared__ int si[32];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const bool first = ps.flags[0] == 0;
  const bool still = !first && ps.flags[4] == 0;  // the last update found no center's members changed
  const int state = ps.flags[7];
  bool stale = ps.wait > 0;  // else prune_dirty_kernel keeps the labels of an untested iteration
  int wait = 0, back = 0;
  if (!first) {
    wait = (state >> 8) & 0xff;
    back = (state >> 16) & 0xff;
    if (!(state & 1)) {  // the last iteration was tested
      stale = ps.flags[1] > ps.cap && (state & 2);
      if (ps.flags[1] <= ps.cap) back = 0;
      else wait = back = min(2 * back + 1, ps.wait);
    }
  }
  const bool full = first || (wait > 0 && !still);
  if (full && !first) --wait;
  float b1 = 0.0f, b2 = 0.0f;
  int i1 = -1;
  for (int j = threadIdx.x; j < ps.k; j += blockDim.x) {
    const float v = ps.shift[j];
    if (v > b1) {
      b2 = b1;
      b1 = v;
      i1 = j;
    } else {
      b2 = fmaxf(b2, v);
    }
    ps.dirty[j] = full;
  }
  auto merge = [&](float o1, float o2, int oi) {
    b2 = fmaxf(fminf(b1, o1), fmaxf(b2, o2));
    if (o1 > b1) {
      b1 = o1;
      i1 = oi;
    }
  };
  for (int o = 16; o > 0; o >>= 1)
    merge(__shfl_down_sync(0xffffffffu, b1, o), __shfl_down_sync(0xffffffffu, b2, o),
          __shfl_down_sync(0xffffffffu, i1, o));
  if (lane == 0) {
    s1[w] = b1;
    s2[w] = b2;
    si[w] = i1;
  }
  __syncthreads();
  if (w == 0) {
    b1 = s1[lane];
    b2 = s2[lane];
    i1 = si[lane];
    for (int o = 16; o > 0; o >>= 1)
      merge(__shfl_down_sync(0xffffffffu, b1, o), __shfl_down_sync(0xffffffffu, b2, o),
            __shfl_down_sync(0xffffffffu, i1, o));
    if (lane == 0) {
      ps.top[0] = b1;
      ps.top[1] = b2;
      ps.flags[0] = 1;
      ps.flags[1] = full ? 0x7fffffff : 0;
      ps.flags[2] = 0;  // the scan of the centers counts from zero
      ps.flags[3] = i1;
      ps.flags[4] = full;
      ps.flags[5] = still;  // no center has moved: every label and bound stands and nothing is scanned
      ps.flags[6] = full || still ? 0 : ps.k;
      ps.flags[7] = (full ? 1 : 0) | (stale ? 2 : 0) | wait << 8 | back << 16;
    }
  }
}

// Moves every row's bounds with the centers and lists the rows they no longer prove. Once more than
// `cap` rows are listed every row will be scanned (and its bounds written anew): the blocks still
// to come return. Where lab_old is stale it takes the labels of the last update on the way.
__global__ void __launch_bounds__(PF_THREADS)
prune_filter_kernel(PruneState ps, const int* labels, const int* stop) {
  if (grid_enter()) return;
  if (stopped(stop)) return;
  __shared__ int wsum[PF_THREADS / 32];
  __shared__ int base_sh;
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  if (ps.flags[5]) return;
  const float top1 = ps.top[0], top2 = ps.top[1];
  const int topi = ps.flags[3];
  const bool stale = ps.flags[7] & 2;
  for (long long b0 = (long long)blockIdx.x * PF_ROWS; b0 < ps.n; b0 += (long long)gridDim.x * PF_ROWS) {
    if (threadIdx.x == 0) base_sh = *(volatile int*)(ps.flags + 1);
    __syncthreads();
    if (base_sh > ps.cap) return;  // uniform over the block
    const long long i0 = b0 + 4 * threadIdx.x;
    float u[4], l[4];
    int a[4];
    if (i0 + 4 <= ps.n) {
      const float4 uv = *reinterpret_cast<const float4*>(ps.ub + i0);
      const float4 lv = *reinterpret_cast<const float4*>(ps.lb + i0);
      const int4 av = *reinterpret_cast<const int4*>(labels + i0);
      u[0] = uv.x, u[1] = uv.y, u[2] = uv.z, u[3] = uv.w;
      l[0] = lv.x, l[1] = lv.y, l[2] = lv.z, l[3] = lv.w;
      a[0] = av.x, a[1] = av.y, a[2] = av.z, a[3] = av.w;
    } else {
#pragma unroll
      for (int r = 0; r < 4; ++r) {
        const bool in = i0 + r < ps.n;
        u[r] = in ? ps.ub[i0 + r] : 0.0f;
        l[r] = in ? ps.lb[i0 + r] : 0.0f;
        a[r] = in ? labels[i0 + r] : 0;
      }
    }
    unsigned fail = 0;
#pragma unroll
    for (int r = 0; r < 4; ++r) {
      if (i0 + r >= ps.n) continue;
      const bool lab_ok = a[r] >= 0 && a[r] < ps.k;  // always, but for an error upstream
      const float sh = lab_ok ? ld(ps.shift + a[r]) : -1.0f;
      const float near = lab_ok ? ld(ps.clb + a[r]) : 0.0f;
      u[r] = sh < 0.0f ? INFINITY : __fadd_ru(u[r], sh);
      l[r] = __fsub_rd(l[r], a[r] == topi ? top2 : top1);
      // the nearest other center is at least `near` from this one, hence near - ub from the row;
      // a NaN (inf - inf) fails the comparison below
      const float l2 = __fsub_rd(near, u[r]);
      l[r] = l2 > l[r] ? l2 : l[r];
      // 2^-20 covers the rounding of the FP64 distances the label is defined by
      if (!(__fmul_ru(u[r], 1.0f + 0x1p-20f) < l[r])) fail |= 1u << r;
    }
    if (i0 + 4 <= ps.n) {
      *reinterpret_cast<float4*>(ps.ub + i0) = make_float4(u[0], u[1], u[2], u[3]);
      *reinterpret_cast<float4*>(ps.lb + i0) = make_float4(l[0], l[1], l[2], l[3]);
      if (stale) *reinterpret_cast<int4*>(ps.lab_old + i0) = make_int4(a[0], a[1], a[2], a[3]);
    } else {
      for (int r = 0; r < 4; ++r)
        if (i0 + r < ps.n) {
          ps.ub[i0 + r] = u[r];
          ps.lb[i0 + r] = l[r];
          if (stale) ps.lab_old[i0 + r] = a[r];
        }
    }
    // one block-wide scan and one atomic per block step
    const int c = __popc(fail);
    int inc = c;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int t = __shfl_up_sync(0xffffffffu, inc, o);
      if (lane >= o) inc += t;
    }
    if (lane == 31) wsum[w] = inc;
    __syncthreads();
    if (threadIdx.x == 0) {
      int t = 0;
      for (int v = 0; v < PF_THREADS / 32; ++v) {
        const int x = wsum[v];
        wsum[v] = t;
        t += x;
      }
      base_sh = t ? atomicAdd(ps.flags + 1, t) : 0;
    }
    __syncthreads();
    int at = base_sh + wsum[w] + inc - c;
#pragma unroll
    for (int r = 0; r < 4; ++r)
      if (fail & (1u << r)) {
        if (at < ps.cap) ps.list[at] = (int)(i0 + r);
        ++at;
      }
    __syncthreads();
  }
}

__global__ void __launch_bounds__(256, 4)
prune_gather_kernel(PruneState ps, const uint4* Xb, const uint4* Xl, int row_vec,
                                    const int* stop) {
  if (grid_enter()) return;
  const int halt = stop ? pinned(stop) : 0;
  const int cnt = pinned(ps.flags + 1);
  if (halt) return;
  if (cnt > ps.cap) return;
  copy_listed_rows(ps.list, cnt, Xb, Xl, row_vec, static_cast<uint4*>(ps.Xc), static_cast<uint4*>(ps.Xlc),
                   ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5,
                   ((long long)gridDim.x * blockDim.x) >> 5, threadIdx.x & 31);
}

// Marks the old and the new center of every scanned row whose label changed since the last update
// (every center, where the rows were not tested or lab_old is not known for all of them; it is kept after an
// untested iteration where none of these may follow another, else by the next filter). A block
// collects its marks in shared memory where the centers fit: in early iterations hundreds of
// thousands of rows mark the same few hundred centers (898,790 rows, K=256: 300 us through global
// memory).
constexpr int kDirtyShared = 32768;

__global__ void __launch_bounds__(1024)
prune_dirty_kernel(PruneState ps, const int* labels, const int* stop) {
  if (grid_enter()) return;
  const int halt = stop ? pinned(stop) : 0;
  const int cnt = pinned(ps.flags + 1), state = pinned(ps.flags + 7);
  if (halt) return;
  if (cnt == 0) return;
  if (state & 1) {  // untested: prune_top_kernel marked every center
    if (state & 2) return;
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < ps.n;
         i += (long long)gridDim.x * blockDim.x)
      ps.lab_old[i] = labels[i];
    return;
  }
  if (cnt > ps.cap && (state & 2)) {  // the filter stopped before lab_old was known for all rows
    for (int j = blockIdx.x * blockDim.x + threadIdx.x; j < ps.k; j += gridDim.x * blockDim.x) {
      ps.dirty[j] = 1;
      ps.flags[4] = 1;
    }
    return;
  }
  extern __shared__ unsigned char mark[];
  const bool sh = ps.k <= kDirtyShared;
  if (sh) {
    for (int j = threadIdx.x; j < ps.k; j += blockDim.x) mark[j] = 0;
    __syncthreads();
  }
  const bool all = cnt > ps.cap;
  const long long total = all ? ps.n : cnt;
  bool changed = false;
  auto set = [&](int j) {
    if (j < 0 || j >= ps.k) return;
    if (sh) mark[j] = 1;
    else if (!*(volatile int*)(ps.dirty + j)) ps.dirty[j] = 1;
  };
#pragma unroll 4
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < total;
       i += (long long)gridDim.x * blockDim.x) {
    const long long pt = all ? i : (long long)ld(ps.list + i);
    const int a = ps.lab_old[pt], b = labels[pt];
    if (a == b) continue;
    ps.lab_old[pt] = b;
    changed = true;
    set(a);
    set(b);
  }
  if (!__syncthreads_or(changed)) return;
  if (threadIdx.x == 0) ps.flags[4] = 1;
  if (sh)
    for (int j = threadIdx.x; j < ps.k; j += blockDim.x)
      if (mark[j]) ps.dirty[j] = 1;
}

// ------------------------------------ batched problems ------------------------------------
// One block per problem: its two largest moves, and its centers' dirty marks cleared (set in the first
// iteration).
__global__ void __launch_bounds__(256)
prune_top_batched_kernel(PruneBatch pb) {
  if (grid_enter()) return;
  __shared__ float s1[8], s2[8];
  __shared__ int si[8];
  const PruneState& ps = pb.ps;
  const int prob = blockIdx.x, lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int first = ps.flags[0] == 0;
  const int c0 = pb.c_off[prob], k = pb.kp[prob];
  float b1 = 0.0f, b2 = 0.0f;
  int i1 = -1;
  auto merge = [&](float o1, float o2, int oi) {
    b2 = fmaxf(fminf(b1, o1), fmaxf(b2, o2));
    if (o1 > b1) {
      b1 = o1;
      i1 = oi;
    }
  };
  for (int j = c0 + threadIdx.x; j < c0 + k; j += blockDim.x) {
    merge(ps.shift[j], 0.0f, j);
    ps.dirty[j] = first;
  }
  for (int o = 16; o > 0; o >>= 1)
    merge(__shfl_down_sync(0xffffffffu, b1, o), __shfl_down_sync(0xffffffffu, b2, o),
          __shfl_down_sync(0xffffffffu, i1, o));
  if (lane == 0) {
    s1[w] = b1;
    s2[w] = b2;
    si[w] = i1;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int v = 1; v < 8; ++v) merge(s1[v], s2[v], si[v]);
    ps.top[2 * prob] = b1;
    ps.top[2 * prob + 1] = b2;
    pb.top_idx[prob] = i1;
  }
}

// One block per window: moves the rows' bounds, then hands the rows they no longer prove to the
// scan -- copied to the compact matrix as ceil(rows / 256) units of their own, or, where most of the
// window fails (or the compact matrix is full), as the window's original units. Units come in any
// order; a window's last one may be part full, which at 4,096 rows a window costs less than a scan
// over all windows' counts would.
__global__ void __launch_bounds__(PF_THREADS)
prune_window_kernel(PruneBatch pb, const int* labels, const uint4* Xb,
                    const uint4* Xl, int row_vec) {
  if (grid_enter()) return;
  constexpr int kPer = kPruneWindow / PF_THREADS;
  __shared__ int rows_sh[kPruneWindow];
  __shared__ int wsum[PF_THREADS / 32];
  __shared__ int unit_sh, crow_sh, total_sh;
  const PruneState& ps = pb.ps;
  const int win = blockIdx.x;
  const int prob = pb.win_prob[win];
  if (pb.done[prob]) return;
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int r0 = pb.win_row[win];
  const int n = (int)min((long long)kPruneWindow, pb.row_end[prob] - r0);
  const bool first = ps.flags[0] == 0;
  unsigned fail = 0;
  if (!first) {
    const float top1 = ps.top[2 * prob], top2 = ps.top[2 * prob + 1];
    const int topi = pb.top_idx[prob];
    const int c0 = pb.c_off[prob], c1 = c0 + pb.kp[prob];
#pragma unroll 4
    for (int i = 0; i < kPer; ++i) {
      const int r = i * PF_THREADS + threadIdx.x;
      if (r >= n) continue;
      const long long pt = (long long)r0 + r;
      const int a = ld(labels + pt);
      const bool lab_ok = a >= c0 && a < c1;
      const float sh = lab_ok ? ld(ps.shift + a) : -1.0f;
      const float near = lab_ok ? ld(ps.clb + a) : 0.0f;
      const float u = sh < 0.0f ? INFINITY : __fadd_ru(ps.ub[pt], sh);
      float l = __fsub_rd(ps.lb[pt], a == topi ? top2 : top1);
      const float l2 = __fsub_rd(near, u);
      l = l2 > l ? l2 : l;
      ps.ub[pt] = u;
      ps.lb[pt] = l;
      if (!(__fmul_ru(u, 1.0f + 0x1p-20f) < l)) fail |= 1u << i;
    }
  }
  const int c = __popc(fail);
  int inc = c;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int t = __shfl_up_sync(0xffffffffu, inc, o);
    if (lane >= o) inc += t;
  }
  if (lane == 31) wsum[w] = inc;
  __syncthreads();
  if (threadIdx.x == 0) {
    int t = 0;
    for (int v = 0; v < PF_THREADS / 32; ++v) {
      const int x = wsum[v];
      wsum[v] = t;
      t += x;
    }
    total_sh = first ? n : t;
    crow_sh = -1;
    if (total_sh > 0) {
      int units = (total_sh + 255) / 256;
      if (!first && total_sh * 5 <= n * 3) {
        const int at = atomicAdd(ps.flags + 4, units * 256);
        if (at + units * 256 <= ps.cap) crow_sh = at;
      }
      if (crow_sh < 0) units = (n + 255) / 256;
      unit_sh = atomicAdd(ps.flags + 3, units);
    }
  }
  __syncthreads();
  const int total = total_sh, crow = crow_sh, unit = unit_sh;
  if (total == 0) return;
  if (crow < 0) {
    for (int u = threadIdx.x; u < (n + 255) / 256; u += PF_THREADS) {
      pb.u_prob[unit + u] = prob;
      pb.u_src[unit + u] = r0 + 256 * u;
      pb.u_cnt[unit + u] = min(256, n - 256 * u);
    }
    return;
  }
  for (int u = threadIdx.x; u < (total + 255) / 256; u += PF_THREADS) {
    pb.u_prob[unit + u] = prob;
    pb.u_src[unit + u] = (crow + 256 * u) | (int)0x80000000;
    pb.u_cnt[unit + u] = min(256, total - 256 * u);
  }
  int at = wsum[w] + inc - c;
#pragma unroll
  for (int i = 0; i < kPer; ++i)
    if (fail & (1u << i)) {
      const int row = r0 + i * PF_THREADS + threadIdx.x;
      rows_sh[at] = row;
      ps.list[crow + at] = row;
      ++at;
    }
  __syncthreads();
  // the rows' planes, 16 bytes per thread at a time
  const int per = row_vec * (Xl ? 2 : 1);
  uint4* Xc = static_cast<uint4*>(ps.Xc);
  uint4* Xlc = static_cast<uint4*>(ps.Xlc);
  constexpr int U = 4;  // loads ahead of their stores
  const int end = total * per;
  for (int e0 = threadIdx.x; e0 < end; e0 += U * PF_THREADS) {
    uint4 x[U];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int e = min(e0 + u * PF_THREADS, end - 1), i = e / per, v = e - i * per;
      const size_t src = (size_t)rows_sh[i] * row_vec;
      x[u] = ld(v < row_vec ? Xb + src + v : Xl + src + (v - row_vec));
    }
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int e = e0 + u * PF_THREADS;
      if (e >= end) break;
      const int i = e / per, v = e - i * per;
      const size_t dst = (size_t)(crow + i) * row_vec;
      *(v < row_vec ? Xc + dst + v : Xlc + dst + (v - row_vec)) = x[u];
    }
  }
}

// The centers that lost or won a row since the last update; one block per window. The scans of this
// iteration are done: block 0 starts the next one's unit table.
__global__ void __launch_bounds__(PF_THREADS)
prune_dirty_batched_kernel(PruneBatch pb, const int* labels) {
  if (grid_enter()) return;
  const PruneState& ps = pb.ps;
  const int win = blockIdx.x;
  if (win == 0 && threadIdx.x == 0) {
    ps.flags[0] = ps.k;
    ps.flags[2] = ps.flags[3] = ps.flags[4] = 0;
  }
  const int prob = pb.win_prob[win];
  if (pb.done[prob]) return;
  const int r0 = pb.win_row[win];
  const int n = (int)min((long long)kPruneWindow, pb.row_end[prob] - r0);
#pragma unroll 4
  for (int r = threadIdx.x; r < n; r += PF_THREADS) {
    const long long pt = (long long)r0 + r;
    const int a = ps.lab_old[pt], b = labels[pt];
    if (a == b) continue;
    ps.lab_old[pt] = b;
    if (a >= 0 && a < ps.k && !*(volatile int*)(ps.dirty + a)) ps.dirty[a] = 1;
    if (b >= 0 && b < ps.k && !*(volatile int*)(ps.dirty + b)) ps.dirty[b] = 1;
  }
}

}  // namespace

bool prune_enabled() {
  const char* v = std::getenv("KMGB_BOUNDS");
  return !(v && std::strcmp(v, "0") == 0);
}

cudaError_t launch_prune_batched(const PruneBatch& pb, const int* labels, const void* Xb,
                                 const void* Xl, long long row_bytes, cudaStream_t s) {
  if (row_bytes % 16 || (Xl && !pb.ps.Xlc)) return cudaErrorInvalidValue;
  launch(prune_top_batched_kernel, (unsigned)pb.P, 256, 0, s)(pb);
  launch(prune_window_kernel, (unsigned)pb.windows, PF_THREADS, 0, s)(
      pb, labels, static_cast<const uint4*>(Xb), static_cast<const uint4*>(Xl), (int)(row_bytes / 16));
  count_launches(2);
  return cudaGetLastError();
}

cudaError_t launch_prune_dirty_batched(const PruneBatch& pb, const int* labels, cudaStream_t s) {
  launch(prune_dirty_batched_kernel, (unsigned)pb.windows, PF_THREADS, 0, s)(pb, labels);
  count_launches(1);
  return cudaGetLastError();
}

cudaError_t launch_prune_dirty(const PruneState& ps, const int* labels, const int* stop,
                               cudaStream_t s) {
  if (inject_fault(kFaultLaunch)) return cudaErrorLaunchOutOfResources;
  const long long blocks = (ps.n + 1023) / 1024, most = 2LL * kmgb::num_sms();
  launch(prune_dirty_kernel, (unsigned)(blocks < most ? blocks : most), 1024,
         ps.k <= kDirtyShared ? ps.k : 0, s)(ps, labels, stop);
  count_launches(1);
  return cudaGetLastError();
}

cudaError_t launch_prune_top(const PruneState& ps, const int* stop, cudaStream_t s) {
  if (inject_fault(kFaultLaunch)) return cudaErrorLaunchOutOfResources;
  launch(prune_top_kernel, 1, 1024, 0, s)(ps, stop);
  count_launches(1);
  return cudaGetLastError();
}

cudaError_t launch_prune_filter(const PruneState& ps, const int* labels, const int* stop,
                                cudaStream_t s) {
  if (inject_fault(kFaultLaunch)) return cudaErrorLaunchOutOfResources;
  const long long steps = (ps.n + PF_ROWS - 1) / PF_ROWS;
  const long long most = kmgb::num_sms() * 8LL;
  launch(prune_filter_kernel, (unsigned)(steps < most ? steps : most), PF_THREADS, 0, s)(ps, labels,
                                                                                     stop);
  count_launches(1);
  return cudaGetLastError();
}

cudaError_t launch_prune_gather(const PruneState& ps, const void* Xb, const void* Xl,
                                long long row_bytes, const int* stop, cudaStream_t s) {
  if (inject_fault(kFaultLaunch)) return cudaErrorLaunchOutOfResources;
  if (row_bytes % 16 || (Xl && !ps.Xlc)) return cudaErrorInvalidValue;
  launch(prune_gather_kernel, kmgb::num_sms() * 4, 256, 0, s)(
      ps, static_cast<const uint4*>(Xb), static_cast<const uint4*>(Xl), (int)(row_bytes / 16), stop);
  count_launches(1);
  return cudaGetLastError();
}

}  // namespace kmgb
