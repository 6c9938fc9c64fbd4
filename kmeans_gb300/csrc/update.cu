// Deterministic center update and SSE for sm_103a.
//
// Replaces the reference's privatised accumulation (main/cuda/ClusterCenters.cu:3-23, one
// G x K x D partial buffer), its per-center reduce and divide (ClusterCenters.cu:47-87), and the
// compactness reduction (main/cuda/Compactness.cu:3-59). Instead of G*K*D partials:
//   1. hist     per-tile label histogram (tile = `tile_pts` consecutive points: 4096 or more, down to
//               512 on small data sets), K x T int32, counted in shared memory (global atomics per
//               peer group when K does not fit);
//   2. scan     exclusive scan of the K-major histogram = start of every (label, tile) run (few
//               counters: by the histogram's last block);
//   3. scatter  eight warps share a tile: each counts its slice, a scan across the warps gives
//               each its first positions, and each walks its points in order writing every
//               point id to start + rank (rank among equal labels of a 32-point step, from
//               ballot peer groups), so the sort by label is stable (ascending point id);
//   4. pieces   every label's run is cut into pieces of kSumPiece points; one lane group per
//               piece (a warp, or 32/L pieces per warp when D <= 64) sums its rows in point
//               order (FP32 data: error-free float-float sum turned into FP64 once per piece;
//               FP64 data: FP64) and the warp the rows' FP64 ||x||^2;
//   5. finalize one block per center adds its pieces in order, divides by the count in FP64,
//               rounds once to FP32 (empty cluster: NaN as in ClusterCenters.cu:81, or keep the
//               previous center), and evaluates the cluster's SSE against the new center with
//               Q - 2 mu.S + n ||mu||^2 in FP64; the last block adds the K cluster SSEs in a fixed
//               order (batched problems and host-streamed tiles: kernels of their own).
// No floating-point atomics: the result is bit-identical run to run and equals the oracle's
// canonical FP64 order.
#include <algorithm>
#include <cfloat>

#include "common.cuh"
#include "kernels.h"

namespace kmgb {
namespace {

constexpr int SCAN_T = 1024;
constexpr int SCAN_V = 8;
constexpr long long SCAN_SEG = SCAN_T * SCAN_V;

__device__ __forceinline__ int warp_incl_scan(int v, int lane) {
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int t = __shfl_up_sync(0xffffffffu, v, o);
    if (lane >= o) v += t;
  }
  return v;
}

// Block-wide exclusive scan of one int per thread (blockDim.x == SCAN_T).
__device__ int block_excl_scan(int v) {
  __shared__ int warp_tot[32];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int inc = warp_incl_scan(v, lane);
  if (lane == 31) warp_tot[w] = inc;
  __syncthreads();
  if (w == 0) {
    const int t = warp_tot[lane];
    const int ti = warp_incl_scan(t, lane);
    warp_tot[lane] = ti - t;
  }
  __syncthreads();
  const int res = warp_tot[w] + inc - v;
  __syncthreads();
  return res;
}

// The run has stopped, or there is nothing to update: no center won or lost a row
// (UpdateWork::any_dirty). Both flags are loaded together.
__device__ __forceinline__ bool skip(const int* stop, const int* any_dirty) {
  const int st = stop ? pinned(stop) : 0;
  const int any = any_dirty ? pinned(any_dirty) : 1;
  return st != 0 || any == 0;
}

// True in every thread of the block that finishes last of the grid (every block calls it once, after
// its writes); *ticket is back at zero afterwards.
__device__ __forceinline__ bool last_block(int* ticket) {
  __shared__ bool last_sh;
  __syncthreads();
  if (threadIdx.x == 0) {
    __threadfence();
    last_sh = atomicAdd(ticket, 1) == (int)gridDim.x - 1;
    if (last_sh) *ticket = 0;
    __threadfence();
  }
  __syncthreads();
  return last_sh;
}

// In-place exclusive scan by one block of SCAN_T threads, of values that other blocks wrote.
__device__ void block_scan_inplace(int* data, long long n) {
  __shared__ int carry_sh;
  int carry = 0;
  for (long long b0 = 0; b0 < n; b0 += SCAN_SEG) {
    const long long base = b0 + (long long)threadIdx.x * SCAN_V;
    int vals[SCAN_V];
    int s = 0;
#pragma unroll
    for (int v = 0; v < SCAN_V; ++v) vals[v] = base + v < n ? __ldcg(data + base + v) : 0;
#pragma unroll
    for (int v = 0; v < SCAN_V; ++v) s += vals[v];
    int pre = block_excl_scan(s) + carry;
#pragma unroll
    for (int v = 0; v < SCAN_V; ++v) {
      if (base + v < n) data[base + v] = pre;
      pre += vals[v];
    }
    if (threadIdx.x == SCAN_T - 1) carry_sh = pre;
    __syncthreads();
    carry = carry_sh;
    __syncthreads();
  }
}

// Sums of the segments; the last block turns them into their exclusive scan.
__global__ void scan_reduce_kernel(const int* in, long long n, int* __restrict__ sums,
                                   int* ticket) {
  if (grid_enter()) return;
  const long long base = (long long)blockIdx.x * SCAN_SEG + (long long)threadIdx.x * SCAN_V;
  int s = 0;
#pragma unroll
  for (int v = 0; v < SCAN_V; ++v)
    if (base + v < n) s += in[base + v];
  __shared__ int red[32];
  for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = s;
  __syncthreads();
  if (threadIdx.x < 32) {
    int t = red[threadIdx.x];
    for (int o = 16; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
    if (threadIdx.x == 0) sums[blockIdx.x] = t;
  }
  if (last_block(ticket)) block_scan_inplace(sums, gridDim.x);
}

// In-place exclusive scan of segment blockIdx.x, plus offset (*offsets)[blockIdx.x] if given.
__global__ void scan_seg_kernel(int* __restrict__ data, long long n, const int* offsets) {
  if (grid_enter()) return;
  const long long base = (long long)blockIdx.x * SCAN_SEG + (long long)threadIdx.x * SCAN_V;
  int vals[SCAN_V];
  int s = 0;
#pragma unroll
  for (int v = 0; v < SCAN_V; ++v) {
    vals[v] = (base + v < n) ? data[base + v] : 0;
    s += vals[v];
  }
  int pre = block_excl_scan(s);
  if (offsets) pre += offsets[blockIdx.x];
#pragma unroll
  for (int v = 0; v < SCAN_V; ++v) {
    if (base + v < n) data[base + v] = pre;
    pre += vals[v];
  }
}

// The counters of one label, tile after tile: their exclusive scan in place by one warp, eight loads in
// flight; returns their sum.
__device__ __forceinline__ int scan_label_row(int* row, int ntiles, int lane) {
  int carry = 0;
  for (int b = 0; b < ntiles; b += 256) {
    int v[8];
#pragma unroll
    for (int u = 0; u < 8; ++u) v[u] = b + 32 * u + lane < ntiles ? row[b + 32 * u + lane] : 0;
#pragma unroll
    for (int u = 0; u < 8; ++u) {
      if (b + 32 * u >= ntiles) break;
      const int inc = warp_incl_scan(v[u], lane);
      if (b + 32 * u + lane < ntiles) row[b + 32 * u + lane] = carry + inc - v[u];
      carry += __shfl_sync(0xffffffffu, inc, 31);
    }
  }
  return carry;
}

// The counters' scan label by label (a warp each): hist becomes a tile's first position among its
// label's rows, and the last block derives the labels' offsets, member counts and first pieces from
// the labels' totals. One launch and one pass over the counters where a scan over all of them took two
// passes and two launches before the offsets' own (256 labels x 220 tiles: 18.8 -> 7.6 us in all).
__global__ void __launch_bounds__(SCAN_T)
label_rows_kernel(int* __restrict__ hist, int k, int ntiles, int* label_off, int* piece_cnt,
                  long long* __restrict__ counts, const int* dirty, int* ticket,
                  const int* any_dirty, const int* stop) {
  if (grid_enter()) return;
  if (skip(stop, any_dirty)) return;
  const int lane = threadIdx.x & 31;
  const int j = (int)blockIdx.x * (SCAN_T / 32) + (int)(threadIdx.x >> 5);
  if (j < k) {
    const int total = scan_label_row(hist + (size_t)j * ntiles, ntiles, lane);
    if (lane == 0) label_off[j] = total;
  }
  if (!last_block(ticket)) return;
  __shared__ int carry_sh[2];
  constexpr int V = 4;
  int carry = 0, pcarry = 0;
  for (int b0 = 0; b0 < k; b0 += SCAN_T * V) {
    const int base = b0 + threadIdx.x * V;
    int c[V], pc[V];
    int s = 0, ps = 0;
#pragma unroll
    for (int v = 0; v < V; ++v) {
      c[v] = base + v < k ? __ldcg(label_off + base + v) : 0;
      pc[v] = base + v >= k || (dirty && !dirty[base + v]) ? 0 : (c[v] + kSumPiece - 1) / kSumPiece;
      s += c[v];
      ps += pc[v];
    }
    int pre = block_excl_scan(s) + carry;
    int ppre = block_excl_scan(ps) + pcarry;
#pragma unroll
    for (int v = 0; v < V; ++v) {
      if (base + v < k) {
        label_off[base + v] = pre;
        piece_cnt[base + v] = ppre;
        if (counts) counts[base + v] = c[v];
      }
      pre += c[v];
      ppre += pc[v];
    }
    if (threadIdx.x == SCAN_T - 1) {
      carry_sh[0] = pre;
      carry_sh[1] = ppre;
    }
    __syncthreads();
    carry = carry_sh[0];
    pcarry = carry_sh[1];
    __syncthreads();
  }
  if (threadIdx.x == 0) {
    label_off[k] = carry;  // (n, but for labels out of range, whose rows are left out)
    piece_cnt[k] = pcarry;
  }
}

// hist[l * ntiles + tile] = members of label l in the tile. SMEM: the tile counts in shared memory (k
// ints) and writes every count; otherwise global atomics per warp group (hist cleared before).
// SMALL (SCAN_T threads): the last block scans the counters and derives the labels' offsets, where
// they are few enough for one block (kSmallHist): one launch instead of three.
constexpr int kSmallHist = 8 * SCAN_T;

template <bool SMEM, bool SMALL>
__global__ void hist_kernel(const int* labels, long long n, int k, int tile_pts,
                            int ntiles, int* __restrict__ hist, int* err, int* label_off,
                            int* piece_cnt, long long* counts, const int* dirty, int* ticket,
                            const int* any_dirty, const int* stop) {
  if (grid_enter()) return;
  if (skip(stop, any_dirty)) return;
  extern __shared__ int cnt_s[];
  const int tile = blockIdx.x;
  const long long i0 = (long long)tile * tile_pts;
  const long long i1 = min(n, i0 + tile_pts);
  const int lane = threadIdx.x & 31;
  if (SMEM) {
    for (int j = threadIdx.x; j < k; j += blockDim.x) cnt_s[j] = 0;
    __syncthreads();
  }
  const int nbits = label_bits(k);
  constexpr int U = SMALL ? 4 : 8;  // labels loaded ahead per thread: one round trip per U steps
  for (long long b = i0; b < i1; b += (long long)blockDim.x * U) {
    int lv[U];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const long long i = b + (long long)u * blockDim.x + threadIdx.x;
      lv[u] = i < i1 ? ld(labels + i) : -1;
    }
#pragma unroll
    for (int u = 0; u < U; ++u) {
      int l = lv[u];
      const long long i = b + (long long)u * blockDim.x + threadIdx.x;
      if (i < i1 && (l < 0 || l >= k)) {
        set_error(err, KMGB_DEV_BAD_LABEL);
        l = -1;
      }
      if (SMEM) {
        if (l >= 0) atomicAdd(&cnt_s[l], 1);
      } else {
        const unsigned peers = warp_peers(l, nbits);
        if (l >= 0 && lane == __ffs(peers) - 1)
          atomicAdd(&hist[(size_t)l * ntiles + tile], __popc(peers));
      }
    }
  }
  if (SMEM) {
    __syncthreads();
    for (int j = threadIdx.x; j < k; j += blockDim.x) hist[(size_t)j * ntiles + tile] = cnt_s[j];
  }
  if (SMALL && last_block(ticket)) {
    // the scan, eight counters a thread, and from its positions in shared memory the labels' offsets,
    // member counts and first pieces (through global memory: three more round trips)
    __shared__ int pos_s[SMALL ? kSmallHist : 1];
    const int total = k * ntiles, t = threadIdx.x;
    int live = t < k && dirty ? ld(dirty + t) : 1;
    int v[8], s = 0;
#pragma unroll
    for (int u = 0; u < 8; ++u) v[u] = 8 * t + u < total ? __ldcg(hist + 8 * t + u) : 0;
#pragma unroll
    for (int u = 0; u < 8; ++u) s += v[u];
    int pre = block_excl_scan(s);
#pragma unroll
    for (int u = 0; u < 8; ++u) {
      if (8 * t + u < total) {
        hist[8 * t + u] = pre;
        pos_s[8 * t + u] = pre;
      }
      pre += v[u];
    }
    __shared__ int carry_sh, all_sh;  // all_sh: the rows with a label (all but labels out of range)
    if (t == SCAN_T - 1) all_sh = pre;
    __syncthreads();
    int carry = 0;
    for (int j0 = 0; j0 < k; j0 += SCAN_T) {
      const int j = j0 + t;
      if (j0 > 0) live = j < k && dirty ? ld(dirty + j) : 1;
      int c = 0, a0 = 0;
      if (j < k) {
        a0 = pos_s[j * ntiles];
        c = (j + 1 < k ? pos_s[(j + 1) * ntiles] : all_sh) - a0;
        label_off[j] = a0;
        if (counts) counts[j] = c;
      }
      const int pc = live ? (c + kSumPiece - 1) / kSumPiece : 0;
      const int first = block_excl_scan(pc) + carry;
      if (j < k) piece_cnt[j] = first;
      if (t == SCAN_T - 1) carry_sh = first + pc;
      __syncthreads();
      carry = carry_sh;
      __syncthreads();
    }
    if (t == 0) {
      label_off[k] = all_sh;
      piece_cnt[k] = carry;
    }
  }
}

// Stable scatter of one tile by one warp, for more labels than scatter_multi_kernel's counters hold.
// SMEM: the tile's first positions are brought to shared memory by the whole block (16,384 labels, 61
// tiles: 91 us with the warp alone, 65 with the block; the rest is the chain of one warp's steps).
constexpr int kScatterLoad = 512;

template <bool SMEM>
__global__ void scatter_kernel(const int* labels, long long n, int k, int tile_pts,
                               int ntiles, int* pos, const int* start,
                               int* __restrict__ sorted, const int* dirty,
                               const int* any_dirty, const int* stop) {
  if (grid_enter()) return;
  if (skip(stop, any_dirty)) return;
  extern __shared__ int cnt_s[];
  const int tile = blockIdx.x;
  const int lane = threadIdx.x;
  if (tile >= ntiles) return;
  if (SMEM) {
    for (int j = threadIdx.x; j < k; j += blockDim.x)
      cnt_s[j] = pos[(size_t)j * ntiles + tile] + (start ? ld(start + j) : 0);
    __syncthreads();
    if (threadIdx.x >= 32) return;
  }
  volatile int* vpos = pos;
  const long long i0 = (long long)tile * tile_pts;
  const long long i1 = min(n, i0 + tile_pts);
  const int nbits = label_bits(k);
  constexpr int U = 8;  // labels loaded ahead: one memory round trip per U steps of 32 points
  for (long long b = i0; b < i1; b += 32 * U) {
    int lv[U];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const long long i = b + 32 * u + lane;
      lv[u] = i < i1 ? ld(labels + i) : -1;
    }
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const long long i = b + 32 * u + lane;
      int l = lv[u];
      if (l < 0 || l >= k || (dirty && !ld(dirty + l))) l = -1;
      const unsigned peers = warp_peers(l, nbits);
      const int leader = __ffs(peers) - 1;
      const int rank = __popc(peers & lanemask_lt());
      int base = 0;
      if (l >= 0 && lane == leader)
        base = SMEM ? cnt_s[l] : vpos[(size_t)l * ntiles + tile];
      base = __shfl_sync(0xffffffffu, base, leader);
      if (l >= 0) sorted[base + rank + (!SMEM && start ? ld(start + l) : 0)] = (int)i;
      if (l >= 0 && lane == leader) {
        const int nv = base + __popc(peers);
        if (SMEM) cnt_s[l] = nv;
        else vpos[(size_t)l * ntiles + tile] = nv;
      }
      __syncwarp();
    }
  }
}

// Stable scatter of one tile by kScatterWarps warps: warp w takes the w-th slice of the tile's
// rows, counts its labels in shared memory, an exclusive scan over the warps (label by label,
// from the tile's start positions) gives every warp its own first positions, and the warps then
// place their rows in parallel. Same positions as one warp walking the tile in order.
constexpr int kScatterWarps = 8;

__global__ void scatter_multi_kernel(const int* labels, long long n, int k,
                                     int tile_pts, int ntiles, const int* pos,
                                     const int* start, int* __restrict__ sorted,
                                     const int* dirty,
                                     const int* any_dirty, const int* stop) {
  if (grid_enter()) return;
  if (skip(stop, any_dirty)) return;
  extern __shared__ int wcnt[];  // [kScatterWarps][k]
  const int tile = blockIdx.x;
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const long long i0 = (long long)tile * tile_pts;
  const long long i1 = min(n, i0 + tile_pts);
  const long long span = ((i1 - i0 + kScatterWarps - 1) / kScatterWarps + 31) / 32 * 32;
  const long long s0 = min(i1, i0 + w * span), s1 = min(i1, s0 + span);
  int* mine = wcnt + (size_t)w * k;
  for (int j = threadIdx.x; j < kScatterWarps * k; j += blockDim.x) wcnt[j] = 0;
  __syncthreads();
  // labels loaded ahead: one memory round trip per U steps of 32 rows, in both passes
  constexpr int U = 8;
  for (long long b = s0; b < s1; b += 32 * U) {
    int lv[U];
#pragma unroll
    for (int u = 0; u < U; ++u) lv[u] = b + 32 * u + lane < s1 ? ld(labels + b + 32 * u + lane) : -1;
#pragma unroll
    for (int u = 0; u < U; ++u)
      if (lv[u] >= 0 && lv[u] < k) atomicAdd(&mine[lv[u]], 1);
  }
  __syncthreads();
  for (int j = threadIdx.x; j < k; j += blockDim.x) {
    int run = pos[(size_t)j * ntiles + tile] + (start ? ld(start + j) : 0);
    for (int v = 0; v < kScatterWarps; ++v) {
      const int c = wcnt[(size_t)v * k + j];
      wcnt[(size_t)v * k + j] = run;
      run += c;
    }
  }
  __syncthreads();
  const int nbits = label_bits(k);
  for (long long b0 = s0; b0 < s1; b0 += 32 * U) {
    int lv[U];
#pragma unroll
    for (int u = 0; u < U; ++u) lv[u] = b0 + 32 * u + lane < s1 ? ld(labels + b0 + 32 * u + lane) : -1;
    if (dirty) {
#pragma unroll
      for (int u = 0; u < U; ++u)
        if (lv[u] >= 0 && lv[u] < k && !ld(dirty + lv[u])) lv[u] = -1;
    }
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const long long i = b0 + 32 * u + lane;
      const int l = lv[u] >= 0 && lv[u] < k ? lv[u] : -1;
      if (!__any_sync(0xffffffffu, l >= 0)) continue;
      const unsigned peers = warp_peers(l, nbits);
      const int leader = __ffs(peers) - 1;
      const int rank = __popc(peers & lanemask_lt());
      int base = 0;
      if (l >= 0 && lane == leader) base = mine[l];
      base = __shfl_sync(0xffffffffu, base, leader);
      if (l >= 0) sorted[base + rank] = (int)i;
      if (l >= 0 && lane == leader) mine[l] = base + __popc(peers);
      __syncwarp();
    }
  }
}

// Piece accumulator. FP32 data: an error-free float-float sum (Knuth's TwoSum on the FP32
// pipe: hi + lo carries ~48 significant bits), turned into one FP64 value per piece; FP64 data:
// a plain FP64 sum (piece_sums_d_kernel). GB300 issues FP64 (and FP32->FP64 conversions) at a small
// fraction of the FP32 rate, so converting every element would bound the update.
struct PieceAcc {
  float hi = 0.0f, lo = 0.0f;
  __device__ __forceinline__ void add(float x) {
    const float t = __fadd_rn(hi, x);
    const float bp = __fsub_rn(t, hi);
    const float err = __fadd_rn(__fsub_rn(hi, __fsub_rn(t, bp)), __fsub_rn(x, bp));
    hi = t;
    lo = __fadd_rn(lo, err);
  }
  __device__ __forceinline__ double value() const { return (double)hi + (double)lo; }
};

// The label of piece p: the last j with pstart[j] <= p (pstart non-decreasing, pstart[0] = 0). The L
// lanes of a group look together, L places at a time (two or three round trips to L2 where a binary
// search takes eight to sixteen); every lane of the warp calls it, p the same within a group.
template <int L>
__device__ __forceinline__ int find_label_group(const int* __restrict__ pstart, int k, int p) {
  const int lane = threadIdx.x & 31, sub = lane % L, shift = lane - sub;
  int lo = 0, n = k;  // the answer lies in [lo, lo + n)
  while (__any_sync(0xffffffffu, n > 1)) {
    const int step = (n + L - 1) / L;
    const int at = lo + sub * step;
    const bool in = n > 1 && sub * step < n && ld(pstart + at) <= p;
    const unsigned bal = (__ballot_sync(0xffffffffu, in) >> shift) & (L == 32 ? 0xffffffffu : (1u << L) - 1u);
    if (n > 1) {
      const int hit = 31 - __clz(bal | 1u);  // place 0 always holds
      n = min(step, n - hit * step);
      lo += hit * step;
    }
  }
  return lo;
}

__device__ __forceinline__ int find_label(const int* __restrict__ pstart, int k, int p) {
  int lo = 0, hi = k - 1;
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if (ld(pstart + mid) <= p) lo = mid;
    else hi = mid - 1;
  }
  return lo;
}

// One warp per piece; dims lane + 32 r in chunks of 256.
__global__ void piece_sums_kernel(const float* X, long long ldx,
                                  const double* qn, const int* sorted,
                                  const int* label_off, const int* pstart,
                                  int k, int d, double* __restrict__ part,
                                  double* __restrict__ partq, const int* any_dirty,
                                  const int* stop) {
  if (grid_enter()) return;
  const int ptot = pinned(pstart + k);
  if (skip(stop, any_dirty)) return;
  const int lane = threadIdx.x & 31;
  const long long gw = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const long long nw = ((long long)gridDim.x * blockDim.x) >> 5;
  for (long long p = gw; p < ptot; p += nw) {
    const int j = find_label(pstart, k, (int)p);
    const int q = (int)p - pstart[j];
    const int b = label_off[j] + q * kSumPiece;
    const int e = min(b + kSumPiece, label_off[j + 1]);
    for (int d0 = 0; d0 < d; d0 += 256) {
      PieceAcc acc[8];
      double qs = 0.0;
#pragma unroll 4
      for (int t = b; t < e; ++t) {
        const int i = ld(sorted + t);
        const float* x = X + (size_t)i * ldx + d0;
#pragma unroll
        for (int r = 0; r < 8; ++r) {
          const int c = lane + 32 * r;
          if (d0 + c < d) acc[r].add(ld(x + c));
        }
        if (qn && d0 == 0) qs += ld(qn + i);
      }
#pragma unroll
      for (int r = 0; r < 8; ++r) {
        const int c = d0 + lane + 32 * r;
        if (c < d) part[(size_t)p * d + c] = acc[r].value();
      }
      if (d0 == 0 && lane == 0 && partq) partq[p] = qs;
    }
  }
}

// FP32 rows with D > 64 whose width and stride are multiples of 4 (16-byte aligned). One warp per
// piece; lane l owns dimensions d0 + 4l .. d0 + 4l + 3 of each 128-dimension chunk d0 of a row.
// The rows travel by cp.async (16 bytes per lane and row) into a per-warp ring of kRingStages
// stages of kRingRows rows in shared memory, so the loads in flight hold no registers: the issuing
// side runs kRingStages - 1 stages ahead of the summing side along the warp's sequence of
// (piece, chunk, 8-row stage), across piece boundaries. A lane reads back only the 16 bytes it
// copied itself, so cp.async.wait_group alone orders its data. Every (piece, dimension) adds the
// piece's points in sorted order with the same float-float TwoSum as the generic kernel, so the
// sums are identical; the piece's sum of ||x||^2 (SSE only) is added as a tree over 32 rows at a
// time.
// Stages are copied and summed whole, zeros past the piece's end: a branch around every row's copy and
// additions, in stages of 8 rows by blocks of four warps, took computeKmeansF on 898,790 x 128, K=256, 50
// iterations 14.07 ms (now 13.80), and 796,160 x 324 15.36 (15.21).
constexpr int kRingStages = 3;
constexpr int kRingRows = 16;
constexpr int kRingWarps = 2;
static_assert(32 % kRingRows == 0, "a stage never straddles a 32-row id window");
static_assert(kRingWarps * kRingStages * kRingRows * 32 * 16 <= 48 * 1024, "static shared memory");

// 16 bytes, of which the first `bytes` (0 or 16) are read and the others zero
__device__ __forceinline__ void cp_async16(uint32_t dst, const void* src, int bytes) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(bytes)
               : "memory");
}
__device__ __forceinline__ void cp_async_commit() {
  asm volatile("cp.async.commit_group;" ::: "memory");
}
template <int N>
__device__ __forceinline__ void cp_async_wait() {
  asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}

// Issuing side of piece_sums_ring_kernel: the cursor over the warp's (piece, chunk, stage)
// sequence. Pieces gw, gw + nw, ...; rows b..e-1 of the current piece, chunk d0, next row t; the
// ids of the 32-row window starting at row wt in `id` (lane l: row wt + l) and, prefetched, of the
// window after it in the same chunk in `id_nx`.
struct RingCursor {
  long long p;
  int b, e, d0, t, wt, id, id_nx;
  double qs;
};

__device__ __forceinline__ int ring_window_id(const int* __restrict__ sorted, int t0, int e,
                                              int lane) {
  return t0 + lane < e ? ld(sorted + t0 + lane) : 0;
}

__device__ __forceinline__ void ring_start_piece(RingCursor& q, long long ptot,
                                                 const int* __restrict__ sorted,
                                                 const int* __restrict__ label_off,
                                                 const int* __restrict__ pstart, int k, int lane) {
  q.d0 = 0;
  q.qs = 0.0;
  if (q.p >= ptot) return;
  const int j = find_label_group<32>(pstart, k, (int)q.p);
  q.b = label_off[j] + ((int)q.p - pstart[j]) * kSumPiece;
  q.e = min(q.b + kSumPiece, label_off[j + 1]);
  q.t = q.b;
  q.id_nx = ring_window_id(sorted, q.b, q.e, lane);
}

// Issues the next stage into ring slot `slot` (one cp.async group, empty once the warp's pieces
// are done) and describes it in `desc`: bit 0 valid, bit 1 last stage of its (piece, chunk),
// bits 8+ chunk; `dp` = its piece.
__device__ __forceinline__ void ring_issue(RingCursor& q, long long ptot, long long nw,
                                           const float* __restrict__ X, long long ldx,
                                           const double* __restrict__ qn,
                                           const int* __restrict__ sorted,
                                           const int* __restrict__ label_off,
                                           const int* __restrict__ pstart, int k, int d,
                                           double* __restrict__ partq, uint32_t slot_addr, int lane,
                                           int& dp, int& desc) {
  if (q.p >= ptot) {
    cp_async_commit();
    dp = 0;
    desc = 0;
    return;
  }
  const bool window = ((q.t - q.b) & 31) == 0;
  double qv = 0.0;
  if (window) {  // a new window: its ids were prefetched; prefetch the next one of the chunk
    q.wt = q.t;
    q.id = q.id_nx;
    q.id_nx = ring_window_id(sorted, q.t + 32, q.e, lane);
    if (qn && q.d0 == 0 && q.t + lane < q.e) qv = ld(qn + q.id);
  }
  const int nr = min(kRingRows, q.e - q.t);
  const int c = q.d0 + 4 * lane;
  const float* xc = X + (c < d ? c : 0);
  const int rows_in = c < d ? nr : 0;
#pragma unroll
  for (int r = 0; r < kRingRows; ++r) {  // rows past the piece: zeros, no branch (their id is a row's)
    const int i = __shfl_sync(0xffffffffu, q.id, (q.t - q.wt + r) & 31);
    cp_async16(slot_addr + r * 512, xc + (size_t)i * ldx, r < rows_in ? 16 : 0);
  }
  cp_async_commit();
  if (window && qn && q.d0 == 0) {  // ||x||^2 of the window's rows: tree sum (FP64)
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) qv += __shfl_xor_sync(0xffffffffu, qv, o);
    q.qs += qv;
  }
  const bool last = q.t + nr >= q.e;
  dp = (int)q.p;
  desc = (q.d0 << 8) | (last ? 2 : 0) | 1;
  q.t += nr;
  if (last) {
    if (q.d0 == 0 && partq && lane == 0) partq[q.p] = q.qs;
    q.d0 += 128;
    if (q.d0 < d) {  // the piece's next chunk: rows from the start again
      q.t = q.b;
      q.id_nx = ring_window_id(sorted, q.b, q.e, lane);
    } else {
      q.p += nw;
      ring_start_piece(q, ptot, sorted, label_off, pstart, k, lane);
    }
  }
}

__global__ void __launch_bounds__(kRingWarps * 32, 4)
piece_sums_ring_kernel(const float* X, long long ldx, const double* qn,
                       const int* sorted, const int* label_off,
                       const int* pstart, int k, int d, double* __restrict__ part,
                       double* __restrict__ partq, const int* any_dirty, const int* stop) {
  if (grid_enter()) return;
  const long long ptot = pinned(pstart + k);
  if (skip(stop, any_dirty)) return;
  __shared__ __align__(16) float4 ring[kRingWarps][kRingStages][kRingRows][32];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const long long nw = (long long)gridDim.x * kRingWarps;
  const uint32_t ring0 = (uint32_t)__cvta_generic_to_shared(&ring[w][0][0][lane]);
  constexpr uint32_t kSlotBytes = kRingRows * 32 * 16;
  static_assert(kRingStages == 3, "the descriptor queue below holds two stages");
  RingCursor q;
  q.p = (long long)blockIdx.x * kRingWarps + w;
  q.b = q.e = q.t = q.wt = q.id = q.id_nx = 0;
  ring_start_piece(q, ptot, sorted, label_off, pstart, k, lane);
  // descriptors of the two stages in flight ahead of the one being issued
  int p0, f0, p1, f1;
  ring_issue(q, ptot, nw, X, ldx, qn, sorted, label_off, pstart, k, d, partq, ring0, lane, p0, f0);
  ring_issue(q, ptot, nw, X, ldx, qn, sorted, label_off, pstart, k, d, partq, ring0 + kSlotBytes,
             lane, p1, f1);
  PieceAcc a0, a1, a2, a3;
  int slot_sum = 0, slot_issue = 2;
  for (;;) {
    int p2, f2;
    ring_issue(q, ptot, nw, X, ldx, qn, sorted, label_off, pstart, k, d, partq,
               ring0 + slot_issue * kSlotBytes, lane, p2, f2);
    cp_async_wait<kRingStages - 1>();  // this lane's copies of stage slot_sum have landed
    if (!(f0 & 1)) break;
    const int c = (f0 >> 8) + 4 * lane;
    {
      const float4* src = &ring[w][slot_sum][0][lane];
#pragma unroll
      for (int r = 0; r < kRingRows; ++r) {  // zeros past the piece change no float-float sum
        const float4 v = src[r * 32];
        a0.add(v.x);
        a1.add(v.y);
        a2.add(v.z);
        a3.add(v.w);
      }
      if ((f0 & 2) && c < d) {
        double* o = part + (size_t)p0 * d + c;
        o[0] = a0.value();
        o[1] = a1.value();
        o[2] = a2.value();
        o[3] = a3.value();
      }
    }
    if (f0 & 2) a0 = a1 = a2 = a3 = PieceAcc{};
    p0 = p1;
    f0 = f1;
    p1 = p2;
    f1 = f2;
    slot_sum = slot_sum == kRingStages - 1 ? 0 : slot_sum + 1;
    slot_issue = slot_issue == kRingStages - 1 ? 0 : slot_issue + 1;
  }
  cp_async_wait<0>();
}

// Small D (a multiple of 4, at most 64): L lanes per piece, each owning 4 consecutive dimensions,
// 32/L pieces per warp. Each lane group walks its own piece's rows in order, so every (piece, dimension)
// float-float sum is the same sequence of additions as in the one-piece-per-warp kernel; the piece's
// sum of ||x||^2 is that kernel's 32-row tree: row i L + sub of a 32-row window is in register i of lane
// sub, so the tree's upper levels join registers and its lower ones lanes. Bound by latency where
// pieces are few (a round trip to L2 costs some 900 cycles): the window's norms and the next window's
// ids are loaded with its rows, and 16 rows are in flight while 16 are summed (6,000 x 32, K=16: an id
// round trip before every 8 rows, the norms piece after piece).
template <int L>
__global__ void __launch_bounds__(128)
piece_sums_small_kernel(const float* X, long long ldx, const double* qn,
                        const int* sorted, const int* label_off,
                        const int* pstart, int k, int d, double* __restrict__ part,
                        double* __restrict__ partq, const int* any_dirty, const int* stop) {
  if (grid_enter()) return;
  const int ptot = pinned(pstart + k);
  if (skip(stop, any_dirty)) return;
  constexpr int G = 32 / L;  // pieces per warp; also ids per lane and window
  constexpr int R = 16;      // rows per batch: one is summed while the next is in flight
  const int lane = threadIdx.x & 31, grp = lane / L, sub = lane % L;
  const long long gw = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const long long nw = ((long long)gridDim.x * blockDim.x) >> 5;
  const int c = 4 * sub;
  for (long long p0 = gw * G; p0 < ptot; p0 += nw * G) {
    const long long p = p0 + grp;
    const bool live = p < ptot;
    const int j = find_label_group<L>(pstart, k, live ? (int)p : 0);
    const int b = live ? ld(label_off + j) + ((int)p - ld(pstart + j)) * kSumPiece : 0;
    const int n = live ? min(kSumPiece, ld(label_off + j + 1) - b) : 0;
    const bool on = live && c < d;
    const float* xc = X + (on ? c : 0);
    auto load_ids = [&](int t, int (&id)[G]) {
#pragma unroll
      for (int i = 0; i < G; ++i)
        id[i] = t + i * L + sub < n ? ld(sorted + b + t + i * L + sub) : -1;
    };
    // rows h .. h + R - 1 of the window whose ids are id (zeros past the piece: adding them changes
    // no float-float sum)
    auto load_rows = [&](const int (&id)[G], int h, float4 (&v)[R]) {
#pragma unroll
      for (int r = 0; r < R; ++r) {
        const int row = __shfl_sync(0xffffffffu, id[(h + r) / L], grp * L + (h + r) % L);
        v[r] = ld(reinterpret_cast<const float4*>(xc + (size_t)max(row, 0) * ldx));  // (no branch)
        if (row < 0) v[r] = make_float4(0.f, 0.f, 0.f, 0.f);
      }
    };
    PieceAcc a0, a1, a2, a3;
    auto add_rows = [&](const float4 (&v)[R]) {
#pragma unroll
      for (int r = 0; r < R; ++r) {
        a0.add(v[r].x);
        a1.add(v[r].y);
        a2.add(v[r].z);
        a3.add(v[r].w);
      }
    };
    double qs = 0.0;
    int id[G], nx[G];
    float4 va[R], vb[R];
    load_ids(0, id);
    load_rows(id, 0, va);
    // the groups' pieces end at different windows: the shuffles take whole warps
    for (int t = 0; __any_sync(0xffffffffu, t < n); t += 32) {
      double q[G];
      load_ids(t + 32, nx);
      load_rows(id, R, vb);
      if (qn) {
#pragma unroll
        for (int i = 0; i < G; ++i) q[i] = id[i] >= 0 ? ld(qn + id[i]) : 0.0;
      }
      add_rows(va);
      load_rows(nx, 0, va);
      add_rows(vb);
      if (qn) {
#pragma unroll
        for (int h = G / 2; h > 0; h >>= 1) {
#pragma unroll
          for (int i = 0; i < h; ++i) q[i] += q[i + h];
        }
#pragma unroll
        for (int o = L / 2; o > 0; o >>= 1) q[0] += __shfl_xor_sync(0xffffffffu, q[0], o);
        if (t < n) qs += q[0];
      }
#pragma unroll
      for (int i = 0; i < G; ++i) id[i] = nx[i];
    }
    if (live && sub == 0 && partq) partq[p] = qs;
    if (on) {
      double* o = part + (size_t)p * d + c;
      o[0] = a0.value();
      o[1] = a1.value();
      o[2] = a2.value();
      o[3] = a3.value();
    }
  }
}

// The same sums where pieces are few: a warp per piece and 32 dimensions, one dimension a lane, every id
// of the piece, then every row in flight at once. A piece is a serial chain of 128 additions, but its
// loads need not be one: with 16 rows ahead a warp waits eight times for L2 (900 cycles each).
__global__ void __launch_bounds__(128)
piece_sums_few_kernel(const float* X, long long ldx, const double* qn,
                      const int* sorted, const int* label_off,
                      const int* pstart, int k, int d, double* __restrict__ part,
                      double* __restrict__ partq, const int* any_dirty, const int* stop) {
  if (grid_enter()) return;
  const int ptot = pinned(pstart + k);
  if (skip(stop, any_dirty)) return;
  constexpr int W = kSumPiece / 32;  // 32-row windows of a piece
  const int groups = (d + 31) / 32;
  const long long total = (long long)ptot * groups;
  const int lane = threadIdx.x & 31;
  const long long gw = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const long long nw = ((long long)gridDim.x * blockDim.x) >> 5;
  for (long long it = gw; it < total; it += nw) {
    const int p = (int)(it / groups), g = (int)(it - (long long)p * groups);
    const int j = find_label_group<32>(pstart, k, p);
    const int b = ld(label_off + j) + (p - ld(pstart + j)) * kSumPiece;
    const int n = min(kSumPiece, ld(label_off + j + 1) - b);
    const int c = g * 32 + lane;
    const bool on = c < d;
    const float* xc = X + (on ? c : 0);
    int id[W];
    double q[W];
#pragma unroll
    for (int w = 0; w < W; ++w) id[w] = 32 * w + lane < n ? ld(sorted + b + 32 * w + lane) : -1;
    float v[kSumPiece];
#pragma unroll
    for (int w = 0; w < W; ++w) {
      q[w] = qn && g == 0 && id[w] >= 0 ? ld(qn + id[w]) : 0.0;
#pragma unroll
      for (int r = 0; r < 32; ++r) {
        const int row = __shfl_sync(0xffffffffu, id[w], r);
        v[32 * w + r] = ld(xc + (size_t)max(row, 0) * ldx);  // (no branch per load)
      }
    }
    PieceAcc a;
#pragma unroll
    for (int w = 0; w < W; ++w) {
      // zeros past the piece: adding them changes no float-float sum (no window ends the loop, or v
      // would be indexed at run time and lie in local memory)
      if (32 * w < n) {
#pragma unroll
        for (int r = 0; r < 32; ++r) a.add(32 * w + r < n ? v[32 * w + r] : 0.0f);
      }
    }
    if (on) part[(size_t)p * d + c] = a.value();
    if (g == 0 && partq) {
      double qs = 0.0;
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) {
#pragma unroll
        for (int w = 0; w < W; ++w) q[w] += __shfl_xor_sync(0xffffffffu, q[w], o);
      }
#pragma unroll
      for (int w = 0; w < W; ++w)
        if (32 * w < n) qs += q[w];
      if (lane == 0) partq[p] = qs;
    }
  }
}

// Canonical piece sums of FP32 rows: the small-D kernel where D <= 64, the cp.async ring kernel
// for other 16-byte-aligned rows, the scalar kernel otherwise.
cudaError_t launch_piece_sums_f32(const float* X, long long ldx, const double* qn,
                                  const int* sorted, const int* label_off, const int* pstart, int k,
                                  int d, double* part, double* partq, const int* any,
                                  const int* stop, long long max_pieces, cudaStream_t s) {
  // (the ring kernel's stage descriptor holds the chunk offset in 23 bits)
  const bool vec = ldx % 4 == 0 && d % 4 == 0 && d < (1 << 23) &&
                   (reinterpret_cast<uintptr_t>(X) & 15) == 0;
  // up to 8 warps of work an SM, what it holds of the kernel: the latency of a piece's loads is what
  // counts (846 pieces of 32 dimensions 16.7 -> 9.1 us, 63 pieces 16.2 -> 7.2; 958 of 128 dimensions,
  // 25 warps an SM, 14.4 with the ring and 20.7 with this kernel)
  const long long few = max_pieces * ((d + 31) / 32);
  if (few <= kmgb::num_sms() * 8LL) {
    launch(piece_sums_few_kernel, (unsigned)((few + 3) / 4), 128, 0, s)(
        X, ldx, qn, sorted, label_off, pstart, k, d, part, partq, any, stop);
    kmgb::count_launches(1);
    return cudaGetLastError();
  }
  const int lanes = !vec || d > 64 ? 32 : (d <= 16 ? 4 : (d <= 32 ? 8 : 16));
  long long warps = (max_pieces + 32 / lanes - 1) / (32 / lanes);
  if (warps > kmgb::num_sms() * 64LL) warps = kmgb::num_sms() * 64LL;
  const unsigned blocks = (unsigned)((warps * 32 + 255) / 256);
  const unsigned sblocks = (unsigned)((warps * 32 + 127) / 128);
  if (vec && lanes < 32) {
    auto kern = lanes == 4 ? piece_sums_small_kernel<4>
                           : (lanes == 8 ? piece_sums_small_kernel<8> : piece_sums_small_kernel<16>);
    launch(kern, sblocks, 128, 0, s)(X, ldx, qn, sorted, label_off, pstart, k, d, part, partq, any, stop);
  } else if (vec) {
    // four blocks (48 KB of ring each) per SM
    const long long cap = kmgb::num_sms() * 4LL * kRingWarps;
    const long long rw = max_pieces < cap ? max_pieces : cap;
    launch(piece_sums_ring_kernel, (unsigned)((rw + kRingWarps - 1) / kRingWarps), kRingWarps * 32, 0, s)(
        X, ldx, qn, sorted, label_off, pstart, k, d, part, partq, any, stop);
  } else
    launch(piece_sums_kernel, blocks, 256, 0, s)(X, ldx, qn, sorted, label_off, pstart, k, d,
                                                    part, partq, any, stop);
  kmgb::count_launches(1);
  return cudaGetLastError();
}

// FP64 rows: one warp per (piece, chunk of 64 dimensions), two dimensions per lane (16 bytes where
// rows are aligned), 16 rows' loads in flight; the additions per (piece, dimension) are in row order.
// (A warp per piece with 4 rows in flight took 258 us for 400,000 x 64, K=256.)
__global__ void __launch_bounds__(128)
piece_sums_d_kernel(const double* X, long long ldx, const int* sorted,
                    const int* label_off, const int* pstart, int k, int d,
                    bool vec, double* __restrict__ part, const int* stop) {
  if (grid_enter()) return;
  if (stopped(stop)) return;
  const int chunks = (d + 63) / 64;
  const long long total = (long long)pstart[k] * chunks;
  const int lane = threadIdx.x & 31;
  const long long gw = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const long long nw = ((long long)gridDim.x * blockDim.x) >> 5;
  constexpr int U = 16;
  for (long long it = gw; it < total; it += nw) {
    const int p = (int)(it / chunks), ch = (int)(it - (long long)p * chunks);
    const int j = find_label(pstart, k, p);
    const int b = label_off[j] + (p - pstart[j]) * kSumPiece;
    const int e = min(b + kSumPiece, label_off[j + 1]);
    const int c = ch * 64 + 2 * lane;
    const bool on0 = c < d, on1 = c + 1 < d;
    double s0 = 0.0, s1 = 0.0;
    for (int t0 = b; t0 < e; t0 += 32) {
      const int ids = t0 + lane < e ? ld(sorted + t0 + lane) : 0;
#pragma unroll
      for (int h = 0; h < 32; h += U) {
        double2 v[U];
#pragma unroll
        for (int r = 0; r < U; ++r) {
          const int i = __shfl_sync(0xffffffffu, ids, h + r);
          v[r] = make_double2(0.0, 0.0);
          if (t0 + h + r < e) {
            const double* x = X + (size_t)i * ldx + c;
            if (vec && on1) {
              v[r] = ld(reinterpret_cast<const double2*>(x));
            } else {
              if (on0) v[r].x = ld(x);
              if (on1) v[r].y = ld(x + 1);
            }
          }
        }
#pragma unroll
        for (int r = 0; r < U; ++r)
          if (t0 + h + r < e) {
            s0 += v[r].x;
            s1 += v[r].y;
          }
      }
    }
    if (on0) part[(size_t)p * d + c] = s0;
    if (on1) part[(size_t)p * d + c + 1] = s1;
  }
}

cudaError_t launch_piece_sums(const float* X, long long ldx, const UpdateWork& w, cudaStream_t s) {
  return launch_piece_sums_f32(X, ldx, nullptr, w.sorted, w.label_off, w.piece_cnt, w.k, w.d, w.part,
                               nullptr, nullptr, w.stop, w.max_pieces, s);
}
cudaError_t launch_piece_sums(const double* X, long long ldx, const UpdateWork& w, cudaStream_t s) {
  const bool vec = ldx % 2 == 0 && (reinterpret_cast<uintptr_t>(X) & 15) == 0;
  const long long items = w.max_pieces * ((w.d + 63) / 64);
  const long long most = kmgb::num_sms() * 16LL;
  const long long warps = items < most ? items : most;
  launch(piece_sums_d_kernel, (unsigned)((warps + 3) / 4), 128, 0, s)(
      X, ldx, w.sorted, w.label_off, w.piece_cnt, w.k, w.d, vec, w.part, w.stop);
  kmgb::count_launches(1);
  return cudaGetLastError();
}

// (double)f from its bits: GB300's FP64 pipe, conversions included, takes a warp 16 cycles per
// instruction. A subnormal, infinite or NaN f is converted there.
__device__ __forceinline__ double widen(float f) {
  const unsigned u = __float_as_uint(f), m = u & 0x7fffffffu;
  if (m - 0x00800000u >= 0x7f000000u && m != 0) return (double)f;
  const unsigned h = m ? (m >> 3) + 0x38000000u : 0u;
  return __hiloint2double((int)((u & 0x80000000u) | h), (int)(u << 29));
}

// 1 / n by Newton's iteration from the FP32 reciprocal (relative errors 2^-23, 2^-46, 2^-52).
__device__ __forceinline__ double reciprocal_of_count(int n, double nd) {
  double r = widen(__frcp_rn((float)n));
  r = fma(r, fma(-nd, r, 1.0), r);
  return fma(r, fma(-nd, r, 1.0), r);
}

// A center's coordinate: the FP64 quotient s / n rounded to FP32. s times the reciprocal is within 3
// units in the last place of that quotient, so it rounds to the same FP32 number unless it lies within
// 8 of the middle between two; only there, and outside FP32's normal range, the division itself (some
// twenty FP64 instructions) runs.
__device__ __forceinline__ float mean_rn(double s, double nd, double rn) {
  const double q = s * rn;
  const long long b = __double_as_longlong(q);
  const unsigned ex = (unsigned)(b >> 52) & 0x7ffu, low = (unsigned)b & 0x1fffffffu;
  if ((b << 1) == 0) return __int_as_float((int)(b >> 32));  // a zero of s's sign
  if (ex - 897u > 252u || low - 0x0ffffff8u <= 16u) return __double2float_rn(__ddiv_rn(s, nd));
  const unsigned m = (unsigned)(b >> 29);  // 23 bits of significand, the exponent above (modulo 512)
  return __uint_as_float(((unsigned)(b >> 32) & 0x80000000u) |
                         (m - (896u << 23) + (low > 0x10000000u ? 1u : 0u)));
}

// Half of a dimension's share n mu^2 - 2 mu s of the SSE identity.
__device__ __forceinline__ double half_sse_share(float mu, double s, double nd) {
  const double m = widen(mu);
  return m * fma(0.5 * nd, m, -s);
}

// A center's piece sums of one dimension (part[p * d], p0 <= p < p1) added in piece order, U loads
// in flight. An addition runs only where there is a piece (the empty statement keeps the compiler from
// running all of them and selecting): the FP64 pipe is what bounds the kernels that call this.
template <int U>
__device__ __forceinline__ double sum_pieces_by(const double* __restrict__ part, int d, int p0, int p1) {
  double s = 0.0;
  for (int p = p0; p < p1; p += U) {
    double v[U];
#pragma unroll
    for (int i = 0; i < U; ++i)
      if (p + i < p1) v[i] = ld(part + (size_t)(p + i) * d);
#pragma unroll
    for (int i = 0; i < U; ++i) {
      if (p + i >= p1) break;
      asm volatile("" : "+d"(s));
      s += v[i];
    }
  }
  return s;
}

__device__ __forceinline__ double sum_pieces(const double* __restrict__ part, int d, int p0, int p1) {
  return p1 - p0 <= 4 ? sum_pieces_by<4>(part, d, p0, p1) : sum_pieces_by<16>(part, d, p0, p1);
}

// One warp per (center j, group g of 32 dimensions): lane c of group g owns dimension
// g*32 + c, adds the center's piece sums in piece order (the canonical order: centers are
// unchanged by the split), divides in FP64 and rounds once. The group's SSE term
// sum_c (n mu^2 - 2 mu s) lands in sse_k[j * G + g]; group 0 adds the members' sum of ||x||^2.
__global__ void finalize_kernel(const double* part, const double* partq,
                                const int* label_off, const int* pstart,
                                int k, int d, float* __restrict__ C, long long ldc,
                                int empty_policy, double* __restrict__ sse_k,
                                const int* dirty, const int* stop) {
  if (grid_enter()) return;
  if (stopped(stop)) return;
  const int groups = (d + 31) / 32;
  const long long wid = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int lane = threadIdx.x & 31;
  if (wid >= (long long)k * groups) return;
  const int j = (int)(wid / groups), g = (int)(wid - (long long)j * groups);
  if (dirty && !dirty[j]) return;
  const int c = g * 32 + lane;
  const int n = label_off[j + 1] - label_off[j];
  const int p0 = pstart[j], p1 = pstart[j + 1];
  double sse = 0.0;
  if (c < d) {
    const double s = sum_pieces(part + c, d, p0, p1);
    float mu;
    if (n > 0) {
      const double nd = (double)n;
      mu = mean_rn(s, nd, reciprocal_of_count(n, nd));
      sse = 2.0 * half_sse_share(mu, s, nd);
    } else if (empty_policy == 1) {
      mu = C[(size_t)j * ldc + c];
    } else {
      mu = __int_as_float(0x7fc00000);
    }
    C[(size_t)j * ldc + c] = mu;
  }
  for (int o = 16; o > 0; o >>= 1) sse += __shfl_xor_sync(0xffffffffu, sse, o);
  // the members' sum of ||x||^2, in piece order: the warp loads 32 pieces at a time, every
  // lane adds them in order from shuffles
  double q = 0.0;
  if (g == 0 && partq && n > 0 && sse_k) {
    for (int b = p0; b < p1; b += 32) {
      const int cnt = min(32, p1 - b);
      const double v = lane < cnt ? ld(partq + b + lane) : 0.0;
      for (int i = 0; i < cnt; ++i) q += __shfl_sync(0xffffffffu, v, i);
    }
  }
  if (lane == 0 && sse_k) sse_k[(size_t)j * groups + g] = (n > 0) ? sse + q : 0.0;
}

// Clusters whose identity SSE (Q - 2 mu.S + n |mu|^2, summed over the groups) is within
// 1e-9 Q of zero -- singletons, duplicates, variance far below the magnitude of the points --
// get their SSE again in the direct form sum_i sum_d ((double)x - (double)mu)^2 over the
// members (exactly 0 when every member equals the center, as the reference's compactness,
// Compactness.cu:3-59, gives); the identity's cancellation error is of the order of 1e-15 Q.
// One warp per center; the direct sum only runs for flagged clusters.
__global__ void sse_fixup_kernel(double* __restrict__ sse_k, int groups,
                                 const double* partq, const int* label_off,
                                 const int* pstart, int k, int d,
                                 const float* X, long long ldx,
                                 const int* sorted, const float* C,
                                 long long ldc, const int* dirty, const int* stop) {
  if (grid_enter()) return;
  if (stopped(stop)) return;
  const long long wid = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int lane = threadIdx.x & 31;
  if (wid >= k) return;
  const int j = (int)wid;
  if (dirty && !dirty[j]) return;
  const int m0 = label_off[j], m1 = label_off[j + 1];
  if (m1 <= m0) return;
  double t = 0.0, q = 0.0;
  for (int g = lane; g < groups; g += 32) t += sse_k[(size_t)j * groups + g];
  for (int p = pstart[j] + lane; p < pstart[j + 1]; p += 32) q += partq[p];
  for (int o = 16; o > 0; o >>= 1) {
    t += __shfl_xor_sync(0xffffffffu, t, o);
    q += __shfl_xor_sync(0xffffffffu, q, o);
  }
  if (!(fabs(t) <= 1e-9 * q)) return;
  const float* mu = C + (size_t)j * ldc;
  double s = 0.0;
  for (int m = m0; m < m1; ++m) {
    const float* x = X + (size_t)sorted[m] * ldx;
    for (int c = lane; c < d; c += 32) {
      const double u = (double)x[c] - (double)mu[c];
      s = fma(u, u, s);
    }
  }
  for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
  for (int g = lane; g < groups; g += 32) sse_k[(size_t)j * groups + g] = (g == 0) ? s : 0.0;
}

// The iteration's SSE and the loop's stop rule (kmeans.cpp:1234-1237,1194): relErr = |SSE - SSE_old| /
// |SSE|; the run stops once !(relErr > criterion), NaN included.
// Its inputs are loaded with the caller's first loads (load_loop): one after the other between the
// stores they cost three round trips.
struct LoopIn {
  int it = 0;
  double prev = 0.0, criterion = 0.0;
};
__device__ __forceinline__ LoopIn load_loop(const int* iters_done, const double* sse_prev,
                                            const double* criterion) {
  LoopIn l;
  if (iters_done) l.it = *iters_done;
  if (sse_prev) {
    l.prev = *sse_prev;
    l.criterion = *criterion;
  }
  return l;
}
__device__ __forceinline__ void store_sse(double sse, const LoopIn& l, double* out, int* stop,
                                          double* sse_prev, double* rel_out, int* iters_done,
                                          int indexed) {
  if (indexed && iters_done) out[l.it] = sse;
  else *out = sse;
  if (sse_prev) {
    const double rel = fabs(sse - l.prev) / fabs(sse);
    *sse_prev = sse;
    *rel_out = rel;
    *iters_done = l.it + 1;
    if (stop && !(rel > l.criterion)) *stop = 1;
  }
}

// The single-problem update's last step, a block per center and step, a warp per group of 32 dimensions:
// the center as in finalize_kernel, and its SSE with the cancelled clusters' direct form as in
// sse_fixup_kernel; then the last block adds the centers' terms (strided chains, a tree) and evaluates
// the stop rule as sse_reduce_kernel does: one launch instead of three. Bound by the latency of its
// chain of loads where centers are few, so what does not depend on each other is loaded together
// (64 x 32: 12.0 -> 10.0 us; 256 x 128: 12.2 -> 10.4), and by the FP64 pipe (2 lanes a cycle) where they
// are many, so the lanes' terms meet in shared memory, a block runs one tree for them and one for the
// norms, quotients avoid the division and a block takes several centers before its fence and ticket
// (16,384 x 256: 268 -> 192 us).
__global__ void __launch_bounds__(256)
finalize_update_kernel(const float* X, float* __restrict__ C, long long ldc,
                       int empty_policy, UpdateWork w, double* __restrict__ sse_out) {
  if (grid_enter()) return;
  const int halt = w.stop ? pinned(w.stop) : 0;
  __shared__ double red[256];
  const int lane = threadIdx.x & 31, wp = threadIdx.x >> 5, warps = blockDim.x >> 5;
  const int d = w.d;
  const int groups = (d + 31) / 32;
  LoopIn loop;  // (written by the last block only, at its end)
  if (threadIdx.x == 0) loop = load_loop(w.iters_done, w.sse_prev, w.criterion);
  for (int j = blockIdx.x; j < w.k; j += gridDim.x) {
    const int live = w.dirty ? pinned(w.dirty + j) : 1;  // uniform over the block
    const int m0 = pinned(w.label_off + j), m1 = pinned(w.label_off + j + 1);
    const int p0 = pinned(w.piece_cnt + j), p1 = pinned(w.piece_cnt + j + 1);
    if (halt) return;
    if (!live) continue;
    // the members' sum of ||x||^2: the last warp's lanes over the pieces, the first ones ahead
    double q = 0.0;
    if (wp == warps - 1 && p0 + lane < p1) q = ld(w.partq + p0 + lane);
    const int n = m1 - m0;
    const double nd = (double)n, rn = reciprocal_of_count(n > 0 ? n : 1, nd);
    double half = 0.0;  // of the lane's share of n mu^2 - 2 mu s
    for (int g = wp; g < groups; g += warps) {
      const int c = g * 32 + lane;
      if (c >= d) continue;
      const double s = sum_pieces(w.part + c, d, p0, p1);
      float mu;
      if (n > 0) {
        mu = mean_rn(s, nd, rn);
        half += half_sse_share(mu, s, nd);
      } else if (empty_policy == 1) {
        mu = C[(size_t)j * ldc + c];
      } else {
        mu = __int_as_float(0x7fc00000);
      }
      C[(size_t)j * ldc + c] = mu;
    }
    red[threadIdx.x] = half;
    if (wp == warps - 1)
      for (int p = p0 + 32 + lane; p < p1; p += 32) q += ld(w.partq + p);
    __syncthreads();  // and the center's dimensions are written
    if (wp == warps - 1) {
      double t = 0.0;
      for (int i = 0; i < warps; ++i) t += red[32 * i + lane];
      for (int o = 16; o > 0; o >>= 1) {
        t += __shfl_xor_sync(0xffffffffu, t, o);
        q += __shfl_xor_sync(0xffffffffu, q, o);
      }
      t = fma(2.0, t, q);
      if (n > 0 && fabs(t) <= 1e-9 * q) {
        // cancelled: the direct form (see sse_fixup_kernel)
        const float* mu = C + (size_t)j * ldc;
        t = 0.0;
        for (int m = m0; m < m1; ++m) {
          const float* x = X + (size_t)w.sorted[m] * w.ldx;
          for (int c = lane; c < d; c += 32) {
            const double u = (double)x[c] - (double)mu[c];
            t = fma(u, u, t);
          }
        }
        for (int o = 16; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
      }
      if (lane == 0) w.sse_k[j] = n > 0 ? t : 0.0;
    }
    __syncthreads();  // red serves the next center
  }
  if (!last_block(w.tickets)) return;
  double s = 0.0;
#pragma unroll 4
  for (int i = threadIdx.x; i < w.k; i += blockDim.x) s += __ldcg(w.sse_k + i);
  for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
  if (lane == 0) red[wp] = s;
  __syncthreads();
  if (threadIdx.x == 0) {
    double sse = 0.0;
    for (int i = 0; i < warps; ++i) sse += red[i];
    store_sse(sse, loop, sse_out, w.stop, w.sse_prev, w.rel_out, w.iters_done, w.sse_indexed);
  }
}

// Second level of the SSE reduction plus the loop's stop rule (host-streamed tiles, shards).
__global__ void sse_reduce_kernel(const double* sse_k, int k, double* __restrict__ out,
                                  int* stop, const double* criterion, double* sse_prev,
                                  double* rel_out, int* iters_done, int indexed) {
  if (grid_enter()) return;
  if (stopped(stop)) return;
  __shared__ double red[1024];
  LoopIn loop;
  if (threadIdx.x == 0) loop = load_loop(iters_done, sse_prev, criterion);
  const int per = (k + blockDim.x - 1) / blockDim.x;
  double s = 0.0;
  for (int j = threadIdx.x * per; j < min(k, (int)(threadIdx.x + 1) * per); ++j) s += sse_k[j];
  red[threadIdx.x] = s;
  __syncthreads();
  for (int w = blockDim.x >> 1; w > 0; w >>= 1) {
    if ((int)threadIdx.x < w) red[threadIdx.x] += red[threadIdx.x + w];
    __syncthreads();
  }
  if (threadIdx.x == 0)
    store_sse(red[0], loop, out, stop, sse_prev, rel_out, iters_done, indexed);
}

cudaError_t excl_scan(int* data, long long n, int* tmp, int* ticket, cudaStream_t s) {
  if (n <= 0) return cudaSuccess;
  const long long nb = (n + SCAN_SEG - 1) / SCAN_SEG;
  if (nb > SCAN_SEG) return cudaErrorInvalidValue;
  if (nb > 1) {
    launch(scan_reduce_kernel, (unsigned)nb, SCAN_T, 0, s)(data, n, tmp, ticket);
    kmgb::count_launches(1);
  }
  launch(scan_seg_kernel, (unsigned)nb, SCAN_T, 0, s)(data, n, nb > 1 ? tmp : nullptr);
  kmgb::count_launches(1);
  return cudaGetLastError();
}

}  // namespace

// Tile size of the label histogram: at least 4096 points (the histogram, its scan and the
// scatter's strided counter loads scale with K x T), and K x T below ~16M entries (one scan of
// <= 64 MB).
void plan_update_tiles(long long n, int k, int* tile_pts, int* ntiles) {
  const long long per = (n * (long long)k + (16LL << 20) - 1) / (16LL << 20);
  long long tp = per < 4096 ? 4096 : (per + 31) / 32 * 32;
  if (tp > (1LL << 30)) tp = 1LL << 30;
  *tile_pts = (int)tp;
  *ntiles = (int)((n + tp - 1) / tp);
}

// The same, with smaller tiles where the counters still fit one step of the single-block scan
// (SCAN_SEG): a small data set's histogram and scatter otherwise run on a few SMs (100,000 rows, K=64:
// 25 blocks; scatter 8.2 us). Only for callers whose buffers are sized by this plan.
void plan_update_tiles_fine(long long n, int k, int* tile_pts, int* ntiles) {
  plan_update_tiles(n, k, tile_pts, ntiles);
  while (*tile_pts > 512 && *ntiles < 2 * kmgb::num_sms() &&
         (long long)k * ((n + *tile_pts / 2 - 1) / (*tile_pts / 2)) <= SCAN_SEG)
    *tile_pts /= 2, *ntiles = (int)((n + *tile_pts - 1) / *tile_pts);
}

size_t update_scan_tmp_elems(long long elems) {
  return (size_t)((elems + SCAN_SEG - 1) / SCAN_SEG) + 1;
}

// Stable sort of the point ids by label + per-label offsets and piece starts.
static cudaError_t sort_by_label(const int* labels, const UpdateWork& w, cudaStream_t s) {
  const long long n = w.n;
  const int k = w.k;
  const long long hist_elems = (long long)k * w.ntiles;
  const size_t smem = sizeof(int) * (size_t)k;
  const bool small = hist_elems <= kSmallHist && smem <= 12 * 1024;  // (next to the scan's 32 KB)
  if (small) {
    launch(hist_kernel<true, true>, w.ntiles, SCAN_T, smem, s)(
        labels, n, k, w.tile_pts, w.ntiles, w.hist, w.err, w.label_off, w.piece_cnt, w.counts, w.dirty,
        w.tickets, w.any_dirty, w.stop);
  } else if (smem <= 96 * 1024) {
    if (smem > 48 * 1024)
      KMGB_CUDA_TRY(cudaFuncSetAttribute(hist_kernel<true, false>,
                                         cudaFuncAttributeMaxDynamicSharedMemorySize, 96 * 1024));
    launch(hist_kernel<true, false>, w.ntiles, 256, smem, s)(
        labels, n, k, w.tile_pts, w.ntiles, w.hist, w.err, nullptr, nullptr, nullptr, nullptr, nullptr,
        w.any_dirty, w.stop);
  } else {
    KMGB_CUDA_TRY(cudaMemsetAsync(w.hist, 0, sizeof(int) * hist_elems, s));
    launch(hist_kernel<false, false>, w.ntiles, 256, 0, s)(
        labels, n, k, w.tile_pts, w.ntiles, w.hist, w.err, nullptr, nullptr, nullptr, nullptr, nullptr,
        w.any_dirty, w.stop);
  }
  kmgb::count_launches(1);
  KMGB_CUDA_TRY(cudaGetLastError());
  if (!small) {
    launch(label_rows_kernel, (unsigned)((k + SCAN_T / 32 - 1) / (SCAN_T / 32)), SCAN_T, 0, s)(
        w.hist, k, w.ntiles, w.label_off, w.piece_cnt, w.counts, w.dirty, w.tickets, w.any_dirty,
        w.stop);
    kmgb::count_launches(1);
    KMGB_CUDA_TRY(cudaGetLastError());
  }
  const int* start = small ? nullptr : w.label_off;  // hist counts from there
  const size_t msmem = sizeof(int) * (size_t)k * kScatterWarps;
  if (msmem <= 96 * 1024) {
    if (msmem > 48 * 1024)
      KMGB_CUDA_TRY(cudaFuncSetAttribute(scatter_multi_kernel,
                                         cudaFuncAttributeMaxDynamicSharedMemorySize, 96 * 1024));
    launch(scatter_multi_kernel, w.ntiles, 32 * kScatterWarps, msmem, s)(
        labels, n, k, w.tile_pts, w.ntiles, w.hist, start, w.sorted, w.dirty, w.any_dirty, w.stop);
    kmgb::count_launches(1);
  } else if (smem <= 96 * 1024) {
    if (smem > 48 * 1024)
      KMGB_CUDA_TRY(cudaFuncSetAttribute(scatter_kernel<true>,
                                         cudaFuncAttributeMaxDynamicSharedMemorySize, 96 * 1024));
    launch(scatter_kernel<true>, w.ntiles, kScatterLoad, smem, s)(
        labels, n, k, w.tile_pts, w.ntiles, w.hist, start, w.sorted, w.dirty, w.any_dirty, w.stop);
    kmgb::count_launches(1);
  } else {
    launch(scatter_kernel<false>, w.ntiles, 32, 0, s)(
        labels, n, k, w.tile_pts, w.ntiles, w.hist, start, w.sorted, w.dirty, w.any_dirty, w.stop);
    kmgb::count_launches(1);
  }
  return cudaGetLastError();
}

cudaError_t launch_update(const float* X, const double* qn, const int* labels, float* C,
                          long long ldc, int empty_policy, const UpdateWork& w, double* sse_out,
                          cudaStream_t s) {
  if (inject_fault(kFaultLaunch)) return cudaErrorLaunchOutOfResources;
  const int k = w.k;
  if (w.n <= 0 || k <= 0) return cudaSuccess;
  KMGB_CUDA_TRY(sort_by_label(labels, w, s));
  KMGB_CUDA_TRY(launch_piece_sums_f32(X, w.ldx, qn, w.sorted, w.label_off, w.piece_cnt, k, w.d,
                                     w.part, w.partq, w.any_dirty, w.stop, w.max_pieces, s));
  const int warps = std::min(8, (w.d + 31) / 32);
  if (w.centers_free) KMGB_CUDA_TRY(cudaStreamWaitEvent(s, w.centers_free, 0));
  const int most = kmgb::num_sms() * (64 / warps);  // blocks the SMs hold at a time
  launch(finalize_update_kernel, (unsigned)std::min(k, most), 32 * warps, 0, s)(X, C, ldc, empty_policy, w,
                                                                                sse_out);
  kmgb::count_launches(1);
  return cudaGetLastError();
}

namespace {

// Per-kernel ABI: add this tile's canonical per-center sums to FP64 accumulators. One warp per
// (center, group of 32 dimensions), eight loads in flight, additions in piece order.
__global__ void accumulate_kernel(const double* part, const int* label_off,
                                  const int* pstart, int k, int d,
                                  double* __restrict__ acc, int* __restrict__ acc_counts) {
  if (grid_enter()) return;
  const int groups = (d + 31) / 32;
  const long long wid = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int lane = threadIdx.x & 31;
  if (wid >= (long long)k * groups) return;
  const int j = (int)(wid / groups), g = (int)(wid - (long long)j * groups);
  const int p0 = pstart[j], p1 = pstart[j + 1];
  const int c = g * 32 + lane;
  if (c < d) {
    double s = 0.0;
    int p = p0;
    for (; p + 8 <= p1; p += 8) {
      double v[8];
#pragma unroll
      for (int i = 0; i < 8; ++i) v[i] = ld(part + (size_t)(p + i) * d + c);
#pragma unroll
      for (int i = 0; i < 8; ++i) s += v[i];
    }
    for (; p < p1; ++p) s += ld(part + (size_t)p * d + c);
    acc[(size_t)j * d + c] += s;
  }
  if (g == 0 && lane == 0) acc_counts[j] += label_off[j + 1] - label_off[j];
}

// Host-streamed tiles: add this tile's canonical per-center sums, member counts and sum of
// ||x||^2 to the run's FP64 accumulators (the tile's pieces in piece order, then one addition per
// tile, tiles in order).
__global__ void accumulate_stream_kernel(const double* part,
                                         const double* partq,
                                         const int* label_off,
                                         const int* pstart, int k, int d,
                                         double* __restrict__ accS, int* __restrict__ accN,
                                         double* __restrict__ accQ, const int* stop) {
  if (grid_enter()) return;
  if (stopped(stop)) return;
  const int j = (int)(((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5);
  const int lane = threadIdx.x & 31;
  if (j >= k) return;
  const int p0 = pstart[j], p1 = pstart[j + 1];
  for (int c = lane; c < d; c += 32) {
    double s = 0.0;
    for (int p = p0; p < p1; ++p) s += part[(size_t)p * d + c];
    accS[(size_t)j * d + c] += s;
  }
  if (lane == 0) {
    double q = 0.0;
    for (int p = p0; p < p1; ++p) q += partq[p];
    accQ[j] += q;
    accN[j] += label_off[j + 1] - label_off[j];
  }
}

// Host-streamed tiles: centers and SSE terms from the run's accumulators, one warp per (center,
// group of 32 dimensions) as finalize_kernel.
__global__ void finalize_stream_kernel(const double* accS, const int* accN,
                                       const double* accQ, int k, int d,
                                       float* __restrict__ C, long long ldc, int empty_policy,
                                       double* __restrict__ sse_k, const int* stop) {
  if (grid_enter()) return;
  if (stopped(stop)) return;
  const int groups = (d + 31) / 32;
  const long long wid = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int lane = threadIdx.x & 31;
  if (wid >= (long long)k * groups) return;
  const int j = (int)(wid / groups), g = (int)(wid - (long long)j * groups);
  const int c = g * 32 + lane;
  const long long n = accN[j];
  double sse = 0.0;
  if (c < d) {
    const double s = accS[(size_t)j * d + c];
    float mu;
    if (n > 0) {
      mu = __double2float_rn(__ddiv_rn(s, (double)n));
      const double m = (double)mu;
      sse = fma((double)n * m, m, -2.0 * m * s);
    } else if (empty_policy == 1) {
      mu = C[(size_t)j * ldc + c];
    } else {
      mu = __int_as_float(0x7fc00000);
    }
    C[(size_t)j * ldc + c] = mu;
  }
  for (int o = 16; o > 0; o >>= 1) sse += __shfl_xor_sync(0xffffffffu, sse, o);
  if (lane == 0) sse_k[(size_t)j * groups + g] = (n > 0) ? sse + (g == 0 ? accQ[j] : 0.0) : 0.0;
}

template <typename T>
__global__ void finalize_acc_kernel(const double* acc, const int* acc_counts,
                                    int k, int d, T* __restrict__ centers, int* __restrict__ counts,
                                    const int* dirty) {
  if (grid_enter()) return;
  const long long total = (long long)k * d;
  for (long long e = (long long)blockIdx.x * blockDim.x + threadIdx.x; e < total;
       e += (long long)gridDim.x * blockDim.x) {
    const int j = (int)(e / d);
    if (dirty && !dirty[j]) continue;
    const int n = acc_counts[j];
    T v;
    if (n > 0) {
      const double q = __ddiv_rn(acc[e], (double)n);
      v = (T)q;
    } else {
      v = (T)__longlong_as_double(0x7ff8000000000000LL);
    }
    centers[e] = v;
    if (counts && e % d == 0) counts[j] = n;
  }
}

}  // namespace

template <typename T>
cudaError_t launch_tile_accumulate(const T* X, long long ldx, const int* labels, const UpdateWork& w,
                                   double* acc, int* acc_counts, cudaStream_t s) {
  if (w.n <= 0 || w.k <= 0) return cudaSuccess;
  KMGB_CUDA_TRY(sort_by_label(labels, w, s));
  KMGB_CUDA_TRY(launch_piece_sums(X, ldx, w, s));
  const long long acc_warps = (long long)w.k * ((w.d + 31) / 32);
  launch(accumulate_kernel, (unsigned)((acc_warps * 32 + 255) / 256), 256, 0, s)(
      w.part, w.label_off, w.piece_cnt, w.k, w.d, acc, acc_counts); kmgb::count_launches(1);
  return cudaGetLastError();
}

template <typename T>
cudaError_t launch_finalize_acc(const double* acc, const int* acc_counts, int k, int d, T* centers,
                                int* counts, cudaStream_t s, const int* dirty) {
  launch(finalize_acc_kernel<T>, kmgb::num_sms() * 4, 256, 0, s)(acc, acc_counts, k, d, centers, counts,
                                                             dirty);
  kmgb::count_launches(1);
  return cudaGetLastError();
}

cudaError_t launch_stream_accumulate(const float* X, long long ldx, const double* qn,
                                     const int* labels, const UpdateWork& w, double* accS,
                                     int* accN, double* accQ, cudaStream_t s) {
  if (w.n <= 0 || w.k <= 0) return cudaSuccess;
  KMGB_CUDA_TRY(sort_by_label(labels, w, s));
  KMGB_CUDA_TRY(launch_piece_sums_f32(X, w.ldx, qn, w.sorted, w.label_off, w.piece_cnt, w.k, w.d,
                                     w.part, w.partq, nullptr, w.stop, w.max_pieces, s));
  launch(accumulate_stream_kernel, (unsigned)(((long long)w.k * 32 + 255) / 256), 256, 0, s)(
      w.part, w.partq, w.label_off, w.piece_cnt, w.k, w.d, accS, accN, accQ, w.stop);
  kmgb::count_launches(1);
  return cudaGetLastError();
}

cudaError_t launch_stream_finalize(const double* accS, const int* accN, const double* accQ,
                                   float* C, long long ldc, int empty_policy, const UpdateWork& w,
                                   double* sse_out, cudaStream_t s) {
  const int k = w.k;
  const long long fin_warps = (long long)k * ((w.d + 31) / 32);
  launch(finalize_stream_kernel, (unsigned)((fin_warps * 32 + 255) / 256), 256, 0, s)(
      accS, accN, accQ, k, w.d, C, ldc, empty_policy, w.sse_k, w.stop);
  kmgb::count_launches(1);
  KMGB_CUDA_TRY(cudaGetLastError());
  launch(sse_reduce_kernel, 1, 1024, 0, s)(w.sse_k, (int)fin_warps, sse_out, w.stop, w.criterion,
                                       w.sse_prev, w.rel_out, w.iters_done, w.sse_indexed);
  kmgb::count_launches(1);
  return cudaGetLastError();
}

template cudaError_t launch_tile_accumulate<float>(const float*, long long, const int*,
                                                   const UpdateWork&, double*, int*, cudaStream_t);
template cudaError_t launch_tile_accumulate<double>(const double*, long long, const int*,
                                                    const UpdateWork&, double*, int*, cudaStream_t);
template cudaError_t launch_finalize_acc<float>(const double*, const int*, int, int, float*, int*,
                                                cudaStream_t, const int*);
template cudaError_t launch_finalize_acc<double>(const double*, const int*, int, int, double*, int*,
                                                 cudaStream_t, const int*);

// ---------------------------------------------------------------------------------------
// Batched Lloyd: many problems of one dimension share X (problem p: rows row_beg[p] ..
// row_end[p]-1) and one center matrix (problem p: centers c_off[p] .. c_off[p]+k[p]-1), labels
// being global center indices. The counting sort uses tiles of tile_pts rows that never cross a
// problem; problem p's counters are hist[hoff[p] + j * ntiles[p] + t] (center j, tile t), so the
// exclusive scan of hist in memory order is the stable order by global label, i.e. problem by
// problem, each sorted exactly as a single problem would be. Piece sums and the finalize step
// are the single-problem kernels over all K centers.
namespace {

// SMEM: the tile's counters in shared memory (one global atomic per peer group, label by label, took
// 14.7 us for 1.5M rows in 775 tiles).
template <bool SMEM>
__global__ void hist_batched_kernel(const int* labels, BatchUpdate b,
                                    int* __restrict__ hist, int* err) {
  if (grid_enter()) return;
  extern __shared__ int cnt_s[];
  const long long st = blockIdx.x;
  const int prob = b.stile_prob[st];
  const int tl = b.stile_local[st];
  const long long i0 = b.row_beg[prob] + (long long)tl * b.tile_pts;
  const long long i1 = min(b.row_end[prob], i0 + b.tile_pts);
  const int cb = b.c_off[prob], kp = b.k[prob], nt = b.ntiles[prob];
  int* h = hist + b.hoff[prob];
  const int lane = threadIdx.x & 31;
  const int nbits = label_bits(kp);
  constexpr int U = 8;  // labels in flight per thread
  if (SMEM) {
    for (int j = threadIdx.x; j < kp; j += blockDim.x) cnt_s[j] = 0;
    __syncthreads();
  }
  for (long long base = i0; base < i1; base += (long long)blockDim.x * U) {
    int lv[U];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const long long i = base + (long long)u * blockDim.x + threadIdx.x;
      lv[u] = i < i1 ? ld(labels + i) - cb : -1;
      if (i < i1 && (lv[u] < 0 || lv[u] >= kp)) {
        set_error(err, KMGB_DEV_BAD_LABEL);
        lv[u] = -1;
      }
    }
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int l = lv[u];
      if (SMEM) {
        if (l >= 0) atomicAdd(&cnt_s[l], 1);
      } else {
        const unsigned peers = warp_peers(l, nbits);
        if (l >= 0 && lane == __ffs(peers) - 1) atomicAdd(&h[(size_t)l * nt + tl], __popc(peers));
      }
    }
  }
  if (SMEM) {
    __syncthreads();
    for (int j = threadIdx.x; j < kp; j += blockDim.x) h[(size_t)j * nt + tl] = cnt_s[j];
  }
}

// label_off[g] = first sorted position of global center g (label_off[K] = rows), piece counts
// and member counts, from the scanned counters.
__global__ void label_offsets_batched_kernel(const int* hist, BatchUpdate b,
                                             int* __restrict__ label_off, int* __restrict__ piece_cnt,
                                             long long* __restrict__ counts,
                                             const int* dirty) {
  if (grid_enter()) return;
  const int gc = blockIdx.x * blockDim.x + threadIdx.x;
  if (gc > b.K) return;
  auto start = [&](int c) -> int {
    if (c >= b.K) return (int)b.n_valid;
    const int prob = b.cprob[c];
    return hist[b.hoff[prob] + (size_t)(c - b.c_off[prob]) * b.ntiles[prob]];
  };
  if (gc == b.K) {
    label_off[b.K] = (int)b.n_valid;
    piece_cnt[b.K] = 0;
    return;
  }
  const int a0 = start(gc), a1 = start(gc + 1);
  label_off[gc] = a0;
  piece_cnt[gc] = dirty && !dirty[gc] ? 0 : (a1 - a0 + kSumPiece - 1) / kSumPiece;
  if (counts) counts[gc] = a1 - a0;
}

// One warp per sort tile. SMEM: the tile's k counters live in shared memory (k <= smem_k).
template <bool SMEM>
__global__ void scatter_batched_kernel(const int* labels, BatchUpdate b, int* pos,
                                       int* __restrict__ sorted, const int* dirty) {
  if (grid_enter()) return;
  extern __shared__ int cnt_s[];
  const long long st = blockIdx.x;
  const int prob = b.stile_prob[st];
  const int tl = b.stile_local[st];
  const long long i0 = b.row_beg[prob] + (long long)tl * b.tile_pts;
  const long long i1 = min(b.row_end[prob], i0 + b.tile_pts);
  const int cb = b.c_off[prob], kp = b.k[prob], nt = b.ntiles[prob];
  volatile int* vpos = pos + b.hoff[prob];
  const int lane = threadIdx.x;
  if (SMEM) {
    for (int j = lane; j < kp; j += 32) cnt_s[j] = vpos[(size_t)j * nt + tl];
    __syncwarp();
  }
  const int nbits = label_bits(kp);
  int lnext = (i0 + lane < i1) ? labels[i0 + lane] : 0;
  for (long long base = i0; base < i1; base += 32) {
    const long long i = base + lane;
    int l = -1;
    if (i < i1) {
      l = lnext - cb;
      if (l < 0 || l >= kp || (dirty && !ld(dirty + cb + l))) l = -1;
    }
    if (base + 32 + lane < i1) lnext = labels[base + 32 + lane];  // next batch in flight
    if (!__any_sync(0xffffffffu, l >= 0)) continue;
    const unsigned peers = warp_peers(l, nbits);
    const int leader = __ffs(peers) - 1;
    const int rank = __popc(peers & lanemask_lt());
    int bs = 0;
    if (l >= 0 && lane == leader) bs = SMEM ? cnt_s[l] : vpos[(size_t)l * nt + tl];
    bs = __shfl_sync(0xffffffffu, bs, leader);
    if (l >= 0) sorted[bs + rank] = (int)i;
    if (l >= 0 && lane == leader) {
      if (SMEM) cnt_s[l] = bs + __popc(peers);
      else vpos[(size_t)l * nt + tl] = bs + __popc(peers);
    }
    __syncwarp();
  }
}

// The same by kScatterWarps warps, as scatter_multi_kernel, where their counters fit (kmax <=
// kScatterMultiK): one warp's chain of steps took 29.5 us for 775 tiles of 2048 rows.
constexpr int kScatterMultiK = 48 * 1024 / 4 / kScatterWarps;

__global__ void scatter_batched_multi_kernel(const int* labels, BatchUpdate b,
                                             const int* pos, int* __restrict__ sorted,
                                             const int* dirty) {
  if (grid_enter()) return;
  extern __shared__ int wcnt[];  // [kScatterWarps][kp]
  const long long st = blockIdx.x;
  const int prob = b.stile_prob[st];
  const int tl = b.stile_local[st];
  const long long i0 = b.row_beg[prob] + (long long)tl * b.tile_pts;
  const long long i1 = min(b.row_end[prob], i0 + b.tile_pts);
  const int cb = b.c_off[prob], kp = b.k[prob], nt = b.ntiles[prob];
  const int* h = pos + b.hoff[prob];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const long long span = ((i1 - i0 + kScatterWarps - 1) / kScatterWarps + 31) / 32 * 32;
  const long long s0 = min(i1, i0 + w * span), s1 = min(i1, s0 + span);
  int* mine = wcnt + (size_t)w * kp;
  for (int j = threadIdx.x; j < kScatterWarps * kp; j += blockDim.x) wcnt[j] = 0;
  __syncthreads();
  constexpr int U = 8;  // labels in flight per lane, in both passes
  auto load = [&](long long base, int (&lv)[U]) {
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const long long i = base + 32 * u + lane;
      lv[u] = i < s1 ? ld(labels + i) - cb : -1;
      if (lv[u] >= kp) lv[u] = -1;
    }
  };
  for (long long base = s0; base < s1; base += 32 * U) {
    int lv[U];
    load(base, lv);
#pragma unroll
    for (int u = 0; u < U; ++u)
      if (lv[u] >= 0) atomicAdd(&mine[lv[u]], 1);
  }
  __syncthreads();
  for (int j = threadIdx.x; j < kp; j += blockDim.x) {
    int run = ld(h + (size_t)j * nt + tl);
    for (int v = 0; v < kScatterWarps; ++v) {
      const int c = wcnt[(size_t)v * kp + j];
      wcnt[(size_t)v * kp + j] = run;
      run += c;
    }
  }
  __syncthreads();
  const int nbits = label_bits(kp);
  for (long long base = s0; base < s1; base += 32 * U) {
    int lv[U];
    load(base, lv);
    if (dirty) {
#pragma unroll
      for (int u = 0; u < U; ++u)
        if (lv[u] >= 0 && !ld(dirty + cb + lv[u])) lv[u] = -1;
    }
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int l = lv[u];
      if (!__any_sync(0xffffffffu, l >= 0)) continue;
      const unsigned peers = warp_peers(l, nbits);
      const int leader = __ffs(peers) - 1;
      const int rank = __popc(peers & lanemask_lt());
      int at = 0;
      if (l >= 0 && lane == leader) at = mine[l];
      at = __shfl_sync(0xffffffffu, at, leader);
      if (l >= 0) sorted[at + rank] = (int)(base + 32 * u + lane);
      if (l >= 0 && lane == leader) mine[l] = at + __popc(peers);
      __syncwarp();
    }
  }
}

// One warp per problem: SSE = sum of its centers' terms; the reference's stop rule per problem
// (kmeans.cpp:1194-1237). A problem that has stopped keeps its history; its centers are
// recomputed from unchanged labels, which reproduces them bit for bit.
// The problem's SSE history slot is its own count of recorded iterations (a stopped problem
// records nothing more), so every iteration issues the same launch: a CUDA graph replays it.
__global__ void sse_batched_kernel(const double* sse_k, int groups, BatchUpdate b) {
  if (grid_enter()) return;
  const long long wid = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int lane = threadIdx.x & 31;
  if (wid >= b.P) return;
  const int prob = (int)wid;
  if (b.done[prob]) return;
  const long long e0 = (long long)b.c_off[prob] * groups;
  const long long e1 = e0 + (long long)b.k[prob] * groups;
  double s = 0.0;
  for (long long e = e0 + lane; e < e1; e += 32) s += sse_k[e];
  for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
  if (lane == 0) {
    const double rel = fabs(s - b.sse_prev[prob]) / fabs(s);
    b.sse_prev[prob] = s;
    b.rel[prob] = rel;
    const int iter = b.iters[prob];
    if (iter < b.max_iters) b.sse_hist[(size_t)prob * b.max_iters + iter] = s;
    b.iters[prob] = iter + 1;
    if (!(rel > b.criterion)) b.done[prob] = 1;
  }
}

}  // namespace

cudaError_t launch_update_batched(const float* X, long long ldx, int d, const double* qn,
                                  const int* labels, float* C, long long ldc, int empty_policy,
                                  const UpdateWork& w, const BatchUpdate& b, cudaStream_t s) {
  if (b.P <= 0 || b.K <= 0 || b.n_valid <= 0) return cudaSuccess;
  KMGB_CUDA_TRY(cudaMemsetAsync(w.hist, 0, sizeof(int) * b.hist_elems, s));
  if (b.kmax <= 12288)
    launch(hist_batched_kernel<true>, (unsigned)b.stiles, 256, sizeof(int) * (size_t)b.kmax, s)(
        labels, b, w.hist, w.err);
  else
    launch(hist_batched_kernel<false>, (unsigned)b.stiles, 256, 0, s)(labels, b, w.hist, w.err);
  count_launches(1);
  KMGB_CUDA_TRY(cudaGetLastError());
  KMGB_CUDA_TRY(excl_scan(w.hist, b.hist_elems, w.scan_tmp, w.tickets, s));
  launch(label_offsets_batched_kernel, (b.K + 1 + 255) / 256, 256, 0, s)(w.hist, b, w.label_off,
                                                                    w.piece_cnt, w.counts, w.dirty);
  count_launches(1);
  KMGB_CUDA_TRY(cudaGetLastError());
  KMGB_CUDA_TRY(excl_scan(w.piece_cnt, b.K + 1, w.scan_tmp, w.tickets, s));
  if (b.kmax <= kScatterMultiK)
    launch(scatter_batched_multi_kernel, (unsigned)b.stiles, 32 * kScatterWarps,
           sizeof(int) * (size_t)b.kmax * kScatterWarps, s)(labels, b, w.hist, w.sorted, w.dirty);
  else if (b.kmax <= 12288)
    launch(scatter_batched_kernel<true>, (unsigned)b.stiles, 32, sizeof(int) * (size_t)b.kmax, s)(
        labels, b, w.hist, w.sorted, w.dirty);
  else
    launch(scatter_batched_kernel<false>, (unsigned)b.stiles, 32, 0, s)(labels, b, w.hist, w.sorted,
                                                                    w.dirty);
  count_launches(1);
  KMGB_CUDA_TRY(cudaGetLastError());
  KMGB_CUDA_TRY(launch_piece_sums_f32(X, ldx, qn, w.sorted, w.label_off, w.piece_cnt, b.K, d,
                                     w.part, w.partq, nullptr, nullptr, w.max_pieces, s));
  const int groups = (d + 31) / 32;
  const long long fin_warps = (long long)b.K * groups;
  if (w.centers_free) KMGB_CUDA_TRY(cudaStreamWaitEvent(s, w.centers_free, 0));
  launch(finalize_kernel, (unsigned)((fin_warps * 32 + 255) / 256), 256, 0, s)(
      w.part, w.partq, w.label_off, w.piece_cnt, b.K, d, C, ldc, empty_policy, w.sse_k, w.dirty,
      nullptr);
  count_launches(1);
  KMGB_CUDA_TRY(cudaGetLastError());
  launch(sse_fixup_kernel, (unsigned)((b.K * 32LL + 255) / 256), 256, 0, s)(
      w.sse_k, groups, w.partq, w.label_off, w.piece_cnt, b.K, d, X, ldx, w.sorted, C, ldc,
      w.dirty, nullptr);
  count_launches(1);
  KMGB_CUDA_TRY(cudaGetLastError());
  launch(sse_batched_kernel, (unsigned)((b.P * 32LL + 255) / 256), 256, 0, s)(w.sse_k, groups, b);
  count_launches(1);
  return cudaGetLastError();
}

}  // namespace kmgb
