// tree_dev.cu -- the far field's octree and target blocks built on the device,
// the same ones as build_tree's (tree.cpp) cell for cell and block for block.
//
// Sources and targets get the Morton keys of tree.cpp (the same FP64 operations,
// so the same bits; bit 63 marks a target) and are sorted together: a stable
// least-digit radix sort of 8-bit digits with the point's index as payload, which
// breaks ties by index as the host sort does.  The tree follows from the sorted
// keys without a walk:
//   d_i  = first level at which points i - 1 and i lie in different cells,
//   D_i  = deepest level at which point i's cell holds more than `limit` points:
//          the largest level shared by points j and j + limit over the windows
//          [j, j + limit] that contain i,
// so the cells that start at point i are those of levels d_i .. min(D_i, 20) + 1,
// and the split ones those up to min(D_i, 20).  Counting them per level and
// scanning gives every cell its breadth-first index; eight lanes per cell find
// its octants' boundaries by binary search.  Target blocks: each split cell of the
// target tree flags the starts of its packed groups of small children.
//
// Host work per build: two reads of two counts (buffer sizes).  The host build it
// replaces copied every position to the host, sorted there and copied the tree
// back: 8.2 of the 9.4 ms of a far-field velocity call at icosahedral level 6.
#include <algorithm>
#include <cmath>

#include <cuda_runtime.h>

#include "farfield_dev.cuh"
#include "lpm_host.hpp"

namespace lpm {

namespace {

using u64k = unsigned long long;

constexpr int kMaxLevel = 21;        // key digits per axis
constexpr int kSortTile = 2048;      // keys per CTA of a sort pass
constexpr int kSortThreads = 256;
constexpr int kScanTile = 1024;      // positions per CTA of the counting kernels
constexpr int kLevels = kMaxLevel + 1;
constexpr int kBoxBlocks = 304;

struct Points {
  const double* p;  // n points, `stride` doubles apart
  int64_t n;
  int stride;
};

// Per-CTA minima of x, y, z, -x, -y, -z of both sets and of -|x|^2 of the targets.
__global__ void __launch_bounds__(256) k_tree_box(Points s, Points t, double* __restrict__ part) {
  __shared__ double sh[7][8];
  double v[7] = {1e300, 1e300, 1e300, 1e300, 1e300, 1e300, 0.0};
  const int64_t step = int64_t(gridDim.x) * 256;
  for (int64_t i = blockIdx.x * int64_t(256) + threadIdx.x; i < s.n + t.n; i += step) {
    const bool src = i < s.n;
    const double* p = src ? s.p + i * s.stride : t.p + (i - s.n) * t.stride;
    const double x = p[0], y = p[1], z = p[2];
    v[0] = fmin(v[0], x), v[1] = fmin(v[1], y), v[2] = fmin(v[2], z);
    v[3] = fmin(v[3], -x), v[4] = fmin(v[4], -y), v[5] = fmin(v[5], -z);
    if (!src) v[6] = fmin(v[6], -(x * x + y * y + z * z));
  }
#pragma unroll
  for (int k = 0; k < 7; ++k) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v[k] = fmin(v[k], __shfl_xor_sync(0xffffffffu, v[k], o));
    if ((threadIdx.x & 31) == 0) sh[k][threadIdx.x >> 5] = v[k];
  }
  __syncthreads();
  if (threadIdx.x < 7) {
    double m = sh[threadIdx.x][0];
    for (int w = 1; w < 8; ++w) m = fmin(m, sh[threadIdx.x][w]);
    part[blockIdx.x * 8 + threadIdx.x] = m;
  }
}

__device__ __forceinline__ u64k spread3(u64k v) {  // 21 bits -> every third bit
  v &= 0x1fffffULL;
  v = (v | (v << 32)) & 0x1f00000000ffffULL;
  v = (v | (v << 16)) & 0x1f0000ff0000ffULL;
  v = (v | (v << 8)) & 0x100f00f00f00f00fULL;
  v = (v | (v << 4)) & 0x10c30c30c30c30c3ULL;
  v = (v | (v << 2)) & 0x1249249249249249ULL;
  return v;
}

// Keys of tree.cpp's key_of in its bounding cube; target bound for rmax.
__global__ void __launch_bounds__(256) k_tree_keys(Points s, Points t, const double* __restrict__ part,
                                                   int nparts, u64k* __restrict__ keys,
                                                   int* __restrict__ idx, double* __restrict__ r2) {
  __shared__ double box[4];
  if (threadIdx.x < 32) {
    double v[7] = {1e300, 1e300, 1e300, 1e300, 1e300, 1e300, 0.0};
    for (int b = threadIdx.x; b < nparts; b += 32)
#pragma unroll
      for (int k = 0; k < 7; ++k) v[k] = fmin(v[k], part[8 * b + k]);
#pragma unroll
    for (int k = 0; k < 7; ++k)
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) v[k] = fmin(v[k], __shfl_xor_sync(0xffffffffu, v[k], o));
    if (threadIdx.x == 0) {
      double ext = 0.0;
#pragma unroll
      for (int c = 0; c < 3; ++c) ext = fmax(ext, __dsub_rn(-v[3 + c], v[c]));
      ext = __dadd_rn(__dmul_rn(ext, 1 + 1e-9), 1e-12);
      for (int c = 0; c < 3; ++c) box[c] = __dsub_rn(v[c], 1e-12);
      box[3] = __ddiv_rn(double(1 << 21), ext);
      if (blockIdx.x == 0) *r2 = -v[6];
    }
  }
  __syncthreads();
  const int64_t i = blockIdx.x * int64_t(256) + threadIdx.x;
  if (i >= s.n + t.n) return;
  const bool src = i < s.n;
  const double* p = src ? s.p + i * s.stride : t.p + (i - s.n) * t.stride;
  u64k k = src ? 0ull : 1ull << 63;
#pragma unroll
  for (int c = 0; c < 3; ++c) {
    const double q = __dmul_rn(__dsub_rn(p[c], box[c]), box[3]);
    const u64k iq = q <= 0 ? 0ull : min(static_cast<u64k>(q), (1ull << 21) - 1);
    k |= spread3(iq) << (2 - c);
  }
  keys[i] = k;
  idx[i] = int(src ? i : i - s.n);
}

// ---- radix sort pass ---------------------------------------------------------
__global__ void __launch_bounds__(kSortThreads) k_sort_hist(const u64k* __restrict__ keys, int64_t n,
                                                            int shift, int nblk,
                                                            int* __restrict__ hist) {
  __shared__ int h[256];
  h[threadIdx.x] = 0;
  __syncthreads();
  const int64_t base = blockIdx.x * int64_t(kSortTile);
#pragma unroll
  for (int k = 0; k < kSortTile / kSortThreads; ++k) {
    const int64_t i = base + k * kSortThreads + threadIdx.x;
    if (i < n) atomicAdd(&h[int(keys[i] >> shift) & 255], 1);
  }
  __syncthreads();
  hist[threadIdx.x * int64_t(nblk) + blockIdx.x] = h[threadIdx.x];
}

// One warp per row: exclusive scan in place of `len` entries, total to tot[row].
__global__ void __launch_bounds__(256) k_scan_rows(int* __restrict__ rows, int nrows, int len,
                                                   int* __restrict__ tot) {
  const int r = blockIdx.x * 8 + (threadIdx.x >> 5), lane = threadIdx.x & 31;
  if (r >= nrows) return;
  int* row = rows + int64_t(r) * len;
  int carry = 0;
  for (int b = 0; b < len; b += 32) {
    const int v = b + lane < len ? row[b + lane] : 0;
    int x = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int y = __shfl_up_sync(0xffffffffu, x, o);
      if (lane >= o) x += y;
    }
    if (b + lane < len) row[b + lane] = carry + x - v;
    carry += __shfl_sync(0xffffffffu, x, 31);
  }
  if (lane == 0) tot[r] = carry;
}

// Stable scatter of a tile: a warp ranks its 256 consecutive keys 32 at a time
// (equal digits by match_any), the digits' warp offsets and the scanned counts
// place them.
__global__ void __launch_bounds__(kSortThreads) k_sort_scatter(
    const u64k* __restrict__ keys, const int* __restrict__ idx, int64_t n, int shift, int nblk,
    const int* __restrict__ hist, const int* __restrict__ tot, u64k* __restrict__ okeys,
    int* __restrict__ oidx) {
  constexpr int W = kSortThreads / 32, PER = kSortTile / kSortThreads;
  __shared__ int cnt[W][256];
  __shared__ int base[256];
  __shared__ int wsum[W];
  const int t = threadIdx.x, w = t >> 5, lane = t & 31;
#pragma unroll
  for (int k = 0; k < W; ++k) cnt[k][t] = 0;
  // digit bases: exclusive scan of the 256 totals, plus this block's offset
  {
    const int v = tot[t];
    int x = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int y = __shfl_up_sync(0xffffffffu, x, o);
      if (lane >= o) x += y;
    }
    if (lane == 31) wsum[w] = x;
    __syncthreads();
    int pre = 0;
    for (int k = 0; k < w; ++k) pre += wsum[k];
    base[t] = pre + x - v + hist[t * int64_t(nblk) + blockIdx.x];
  }
  __syncthreads();
  const int64_t first = blockIdx.x * int64_t(kSortTile) + w * (32 * PER);
  u64k key[PER];
  int rank[PER];
#pragma unroll
  for (int k = 0; k < PER; ++k) {
    const int64_t i = first + k * 32 + lane;
    const bool in = i < n;
    key[k] = in ? keys[i] : 0ull;
    const int d = in ? int(key[k] >> shift) & 255 : 256;
    const unsigned m = __match_any_sync(0xffffffffu, d);
    const int before = __popc(m & ((1u << lane) - 1u));
    rank[k] = in ? cnt[w][d] + before : 0;
    __syncwarp();
    if (in && before == 0) cnt[w][d] += __popc(m);
    __syncwarp();
  }
  __syncthreads();
  int run = base[t];
#pragma unroll
  for (int k = 0; k < W; ++k) {
    const int c = cnt[k][t];
    cnt[k][t] = run;
    run += c;
  }
  __syncthreads();
#pragma unroll
  for (int k = 0; k < PER; ++k) {
    const int64_t i = first + k * 32 + lane;
    if (i >= n) continue;
    const int pos = cnt[w][int(key[k] >> shift) & 255] + rank[k];
    okeys[pos] = key[k];
    oidx[pos] = idx[i];
  }
}

// ---- cells ----------------------------------------------------------------------
// Deepest level at which two keys lie in the same cell (21: equal keys).
__device__ __forceinline__ int shared_level(u64k a, u64k b) {
  const u64k x = (a ^ b) & ~(1ull << 63);
  return x == 0 ? kMaxLevel : kMaxLevel - 1 - (63 - __clzll((long long)x)) / 3;
}
__device__ __forceinline__ u64k prefix(u64k key, int level) {
  return (key & ~(1ull << 63)) >> (3 * (kMaxLevel - level));
}

// First and last level of the listed cells that start at a point: all cells of the
// source tree, the split ones of the target tree.
struct LevelRange {
  int first, last, split;  // split: last level of the point's split cells
};
__device__ LevelRange level_range(const u64k* __restrict__ k, int64_t n, int64_t i, int limit,
                                  bool only_split, const int8_t* sh) {
  // sh[q]: shared level of points (j, j + limit) with j = block start - limit + q
  LevelRange r;
  r.first = i == 0 ? 0 : shared_level(k[i - 1], k[i]) + 1;
  int D = -1;
  for (int q = 0; q <= limit; ++q) D = max(D, int(sh[q]));
  r.split = min(D, kMaxLevel - 1);
  r.last = only_split ? r.split : r.split + 1;
  return r;
}

// MODE 0 counts the listed cells per level into cnt[level][block]; MODE 1 writes
// them: source cells as (start, level, first child or -1, 0), target split cells as
// (start, level, -, -).
template <int MODE>
__global__ void __launch_bounds__(kScanTile) k_tree_cells(const u64k* __restrict__ k, int64_t n,
                                                          int limit, int only_split, int nblk,
                                                          int* __restrict__ cnt,
                                                          const int* __restrict__ tot,
                                                          int4* __restrict__ cells) {
  __shared__ int8_t sh[kScanTile + kTargetBlock];
  __shared__ int wc[kLevels][kScanTile / 32];
  const int t = threadIdx.x, w = t >> 5, lane = t & 31;
  const int64_t b0 = blockIdx.x * int64_t(kScanTile), i = b0 + t;
  for (int q = t; q < kScanTile + limit; q += kScanTile) {
    const int64_t j = b0 - limit + q;
    sh[q] = j >= 0 && j + limit < n ? int8_t(shared_level(k[j], k[j + limit])) : int8_t(-1);
  }
  __syncthreads();
  LevelRange r{1, 0, 0};
  if (i < n) r = level_range(k, n, i, limit, only_split != 0, sh + t);
  for (int l = 0; l < kLevels; ++l) {
    const unsigned m = __ballot_sync(0xffffffffu, l >= r.first && l <= r.last);
    if (lane == 0) wc[l][w] = __popc(m);
  }
  __syncthreads();
  if (MODE == 0) {
    if (t < kLevels) {
      int c = 0;
      for (int q = 0; q < kScanTile / 32; ++q) c += wc[t][q];
      cnt[t * int64_t(nblk) + blockIdx.x] = c;
    }
    return;
  }
  if (t < kLevels) {
    // index of the block's first cell of this level: cells of the levels
    // above, then of the blocks before
    int run = cnt[t * int64_t(nblk) + blockIdx.x];
    for (int l = 0; l < t; ++l) run += tot[l];
    for (int q = 0; q < kScanTile / 32; ++q) {
      const int c = wc[t][q];
      wc[t][q] = run;
      run += c;
    }
  }
  __syncthreads();
  int prev = -1;  // index of this point's cell one level up
  for (int l = 0; l < kLevels; ++l) {
    const bool has = l >= r.first && l <= r.last;
    const unsigned m = __ballot_sync(0xffffffffu, has);
    if (!has) continue;
    const int id = wc[l][w] + __popc(m & ((1u << lane) - 1u));
    cells[id] = make_int4(int(i), l, -1, 0);
    if (!only_split && prev >= 0 && l - 1 <= r.split) cells[prev].z = id;  // first child
    prev = id;
  }
}

// First position in [lo, n) whose prefix at `level` is at least p.
__device__ __forceinline__ int64_t lower_bound(const u64k* __restrict__ k, int64_t lo, int64_t n,
                                               int level, u64k p) {
  int64_t hi = n;
  while (lo < hi) {
    const int64_t m = (lo + hi) >> 1;
    if (prefix(k[m], level) < p) lo = m + 1;
    else hi = m;
  }
  return lo;
}

// Eight lanes per source cell: its end, and its non-empty octants if it is split.
__global__ void __launch_bounds__(128) k_tree_fill(const u64k* __restrict__ k, int64_t n, int ncells,
                                                   int4* __restrict__ cells) {
  const int64_t g = (blockIdx.x * int64_t(128) + threadIdx.x) >> 3;
  const int c = threadIdx.x & 7;
  const unsigned mask = 0xffu << (threadIdx.x & 24);
  if (g >= ncells) return;
  const int4 v = cells[g];
  const int64_t i = v.x;
  const int level = v.y;
  int64_t b;  // lane c: end of octant c (split), lane 7: end of the cell
  if (v.z >= 0)
    b = lower_bound(k, i, n, level + 1, prefix(k[i], level) * 8 + c + 1);
  else
    b = c == 7 ? lower_bound(k, i, n, level, prefix(k[i], level) + 1) : i;
  const int64_t a = __shfl_up_sync(mask, b, 1, 8);
  const bool some = v.z >= 0 && b > (c == 0 ? i : a);
  const int nch = __popc(__ballot_sync(mask, some) & mask);
  if (c == 7) cells[g] = make_int4(v.x, int(b - i), v.z, nch);
}

// Eight lanes per split cell of the target tree: lane 0 packs consecutive small
// octants into groups of at most kTargetBlock and flags their starts (larger octants
// are split cells themselves; at the last level they are cut every kTargetBlock).
__global__ void __launch_bounds__(128) k_tree_groups(const u64k* __restrict__ k, int64_t n,
                                                     const int4* __restrict__ cells, int ncells,
                                                     uint8_t* __restrict__ flag) {
  const int64_t g = (blockIdx.x * int64_t(128) + threadIdx.x) >> 3;
  const int c = threadIdx.x & 7;
  const unsigned mask = 0xffu << (threadIdx.x & 24);
  if (g >= ncells) return;
  const int4 v = cells[g];
  const int64_t i = v.x;
  const int64_t b = lower_bound(k, i, n, v.y + 1, prefix(k[i], v.y) * 8 + c + 1);
  int64_t e[8];
#pragma unroll
  for (int q = 0; q < 8; ++q) e[q] = __shfl_sync(mask, b, q, 8);
  if (c != 0) return;
  int64_t at = i;
  int fill = -1;  // points of the open group, -1: none
  for (int q = 0; q < 8; ++q) {
    const int64_t m = e[q] - at;
    if (m > kTargetBlock) {
      fill = -1;
      if (v.y + 1 >= kMaxLevel)
        for (int64_t x = at; x < e[q]; x += kTargetBlock) flag[x] = 1;
    } else if (m > 0) {
      if (fill < 0 || fill + m > kTargetBlock) {
        flag[at] = 1;
        fill = 0;
      }
      fill += int(m);
    }
    at = e[q];
  }
}

// Flagged positions: counted per CTA (MODE 0), listed in order (MODE 1).
template <int MODE>
__global__ void __launch_bounds__(kScanTile) k_tree_starts(const uint8_t* __restrict__ flag, int64_t n,
                                                           int* __restrict__ cnt,
                                                           int* __restrict__ start) {
  __shared__ int wc[kScanTile / 32];
  const int64_t i = blockIdx.x * int64_t(kScanTile) + threadIdx.x;
  const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const bool f = i < n && flag[i] != 0;
  const unsigned m = __ballot_sync(0xffffffffu, f);
  if (lane == 0) wc[w] = __popc(m);
  __syncthreads();
  if (MODE == 0) {
    if (threadIdx.x == 0) {
      int c = 0;
      for (int q = 0; q < kScanTile / 32; ++q) c += wc[q];
      cnt[blockIdx.x] = c;
    }
    return;
  }
  int id = cnt[blockIdx.x] + __popc(m & ((1u << lane) - 1u));
  for (int q = 0; q < w; ++q) id += wc[q];
  if (f) start[id] = int(i);
}

__global__ void __launch_bounds__(kTargetBlock) k_tree_slots(const int* __restrict__ idx,
                                                             const int* __restrict__ start,
                                                             int nblocks, int64_t n,
                                                             int* __restrict__ tslot) {
  const int b = blockIdx.x;
  const int64_t i = start[b] + threadIdx.x;
  const int64_t end = b + 1 < nblocks ? start[b + 1] : n;
  tslot[b * int64_t(kTargetBlock) + threadIdx.x] = i < end ? idx[i] : -1;
}

int blocks_of(int64_t n, int per) { return int((n + per - 1) / per); }

}  // namespace

// (at most ntgt / 129 split target cells on each of 21 levels)
size_t tree_build_bytes(int64_t nsrc, int64_t ntgt) {
  const size_t n = size_t(nsrc + ntgt);
  return n * (2 * sizeof(u64k) + 2 * sizeof(int)) + 256 * sizeof(int) * (n / kSortTile + 2) +
         2 * kLevels * sizeof(int) * (n / kScanTile + 4) + size_t(ntgt) * (1 + sizeof(int)) +
         (size_t(ntgt) / 6 + 64) * sizeof(int4) + 8 * kBoxBlocks * sizeof(double) + 8192 + 32 * 256;
}

// The caller has reserved tree_build_bytes() in the context's arena.
void build_tree_device(lpm_context& ctx, FFDevice& d, const double* src, int src_stride, int64_t nsrc,
                       const double* tgt, int tgt_stride, int64_t ntgt, int leaf_max) {
  if (nsrc <= 0) throw Error(LPM_ERR_ARG, "build_tree: no sources");
  if (leaf_max < 1 || leaf_max > kMaxLeaf) throw Error(LPM_ERR_ARG, "build_tree: leaf size out of range");
  cudaStream_t st = ctx.stream;
  Arena& ar = ctx.arena;
  const int64_t n = nsrc + ntgt;
  const Points s{src, nsrc, src_stride}, t{tgt, ntgt, tgt_stride};
  u64k* key[2];
  int* idx[2];
  for (int k = 0; k < 2; ++k) {
    key[k] = static_cast<u64k*>(ar.take(sizeof(u64k) * n));
    idx[k] = static_cast<int*>(ar.take(sizeof(int) * n));
  }
  const int nblk = blocks_of(n, kSortTile);
  int* hist = static_cast<int*>(ar.take(sizeof(int) * 256 * size_t(nblk)));
  int* tot = static_cast<int*>(ar.take(sizeof(int) * 512));
  double* part = static_cast<double*>(ar.take(sizeof(double) * 8 * kBoxBlocks));
  double* r2 = static_cast<double*>(ar.take(sizeof(double)));
  const int nbox = std::min(kBoxBlocks, blocks_of(n, 256));
  k_tree_box<<<nbox, 256, 0, st>>>(s, t, part);
  k_tree_keys<<<blocks_of(n, 256), 256, 0, st>>>(s, t, part, nbox, key[0], idx[0], r2);
  ctx.launches += 2;
  for (int pass = 0; pass < 8; ++pass) {
    const int a = pass & 1;
    k_sort_hist<<<nblk, kSortThreads, 0, st>>>(key[a], n, 8 * pass, nblk, hist);
    k_scan_rows<<<32, 256, 0, st>>>(hist, 256, nblk, tot);
    k_sort_scatter<<<nblk, kSortThreads, 0, st>>>(key[a], idx[a], n, 8 * pass, nblk, hist, tot,
                                                  key[a ^ 1], idx[a ^ 1]);
    ctx.launches += 3;
  }
  const u64k *ks = key[0], *kt = key[0] + nsrc;
  const int *is = idx[0], *it = idx[0] + nsrc;
  // counts per level of the two trees: rows 0..21 of each half
  const int bs = blocks_of(nsrc, kScanTile), bt = std::max(1, blocks_of(ntgt, kScanTile));
  int* cs = static_cast<int*>(ar.take(sizeof(int) * kLevels * size_t(bs)));
  int* ct = static_cast<int*>(ar.take(sizeof(int) * kLevels * size_t(bt)));
  int* tots = tot + 256;
  int* tott = tots + 32;
  k_tree_cells<0><<<bs, kScanTile, 0, st>>>(ks, nsrc, leaf_max, 0, bs, cs, nullptr, nullptr);
  k_scan_rows<<<(kLevels + 7) / 8, 256, 0, st>>>(cs, kLevels, bs, tots);
  LPM_CUDA(cudaMemsetAsync(tott, 0, sizeof(int) * 32, st));
  if (ntgt > 0) {
    k_tree_cells<0><<<bt, kScanTile, 0, st>>>(kt, ntgt, kTargetBlock, 1, bt, ct, nullptr, nullptr);
    k_scan_rows<<<(kLevels + 7) / 8, 256, 0, st>>>(ct, kLevels, bt, tott);
    ctx.launches += 2;
  }
  ctx.launches += 2;
  LPM_CUDA(cudaGetLastError());
  int h[64];
  double hr2 = 0.0;
  LPM_CUDA(cudaMemcpyAsync(h, tots, sizeof(h), cudaMemcpyDeviceToHost, st));
  LPM_CUDA(cudaMemcpyAsync(&hr2, r2, sizeof(hr2), cudaMemcpyDeviceToHost, st));
  LPM_CUDA(cudaStreamSynchronize(st));
  int ncells = 0, nsplit = 0;
  for (int l = 0; l < kLevels; ++l) ncells += h[l], nsplit += h[32 + l];

  d.nsrc = nsrc;
  d.ntgt = ntgt;
  // targets move between tree builds: keep a generous margin
  d.rmax = float(1.1 * std::sqrt(hr2) + 0.1);
  d.grow(d.perm, nsrc);
  d.grow(d.cells, ncells);
  LPM_CUDA(cudaMemcpyAsync(d.perm, is, sizeof(int) * nsrc, cudaMemcpyDeviceToDevice, st));
  k_tree_cells<1><<<bs, kScanTile, 0, st>>>(ks, nsrc, leaf_max, 0, bs, cs, tots, d.cells);
  k_tree_fill<<<blocks_of(int64_t(ncells) * 8, 128), 128, 0, st>>>(ks, nsrc, ncells, d.cells);
  ctx.launches += 2;
  int nblocks = 0;
  if (ntgt > 0) {
    uint8_t* flag = static_cast<uint8_t*>(ar.take(size_t(ntgt)));
    int* start = static_cast<int*>(ar.take(sizeof(int) * size_t(ntgt)));
    LPM_CUDA(cudaMemsetAsync(flag, 0, size_t(ntgt), st));
    if (nsplit > 0) {
      int4* split = static_cast<int4*>(ar.take(sizeof(int4) * size_t(nsplit)));
      k_tree_cells<1><<<bt, kScanTile, 0, st>>>(kt, ntgt, kTargetBlock, 1, bt, ct, tott, split);
      k_tree_groups<<<blocks_of(int64_t(nsplit) * 8, 128), 128, 0, st>>>(kt, ntgt, split, nsplit, flag);
      ctx.launches += 2;
    } else {
      LPM_CUDA(cudaMemsetAsync(flag, 1, 1, st));  // everything in one block
    }
    k_tree_starts<0><<<bt, kScanTile, 0, st>>>(flag, ntgt, ct, nullptr);
    k_scan_rows<<<1, 256, 0, st>>>(ct, 1, bt, tott);
    k_tree_starts<1><<<bt, kScanTile, 0, st>>>(flag, ntgt, ct, start);
    ctx.launches += 3;
    LPM_CUDA(cudaMemcpyAsync(&nblocks, tott, sizeof(int), cudaMemcpyDeviceToHost, st));
    LPM_CUDA(cudaStreamSynchronize(st));
    d.grow(d.tslot, size_t(nblocks) * kTargetBlock);
    k_tree_slots<<<nblocks, kTargetBlock, 0, st>>>(it, start, nblocks, ntgt, d.tslot);
    ctx.launches++;
  }
  d.nblocks = nblocks;
  LPM_CUDA(cudaGetLastError());
  d.grow(d.ys, nsrc);
  d.grow(d.cd, size_t(kCellF) * ncells);
  d.grow(d.xt, size_t(kTargetBlock) * nblocks);
  d.grow(d.box, size_t(nblocks));
  d.grow(d.far, size_t(kFarCap) * nblocks);
  d.grow(d.near, size_t(kNearCap) * nblocks);
  d.grow(d.lrn, size_t(kLearnCap) * nblocks);
  d.grow(d.cnt, size_t(nblocks));
  d.grow(d.counter, 4);
  d.ncells = ncells;  // built
}

}  // namespace lpm
