// farfield.cu -- octree evaluation of the BVE sphere velocity sum.
//
// Per evaluation (all on the context stream, capturable in a CUDA graph):
//   k_ff_sort_src   packed double4_16a sources -> Morton-ordered float4
//   k_ff_cells      per cell: centre, radius, frame, moments to order 4
//                   (FP32 per batch, FP64 across batches and threads)
//   k_ff_tblocks    per block of 128 Morton-ordered targets: centre, radius
//   k_ff_lists      a warp per target block: tree walk with the opening criterion
//                   h <= theta (D - r_b): far cells (of >= kExactMax points;
//                   smaller accepted cells are leaves and join the near
//                   list), near leaves, and the far cells close enough
//                   (h / (D - r_b) >= rho_min) for the learned correction; a
//                   block whose lists overflow is marked for the direct sum
//   k_ff_eval       per target block and part: exact FP32 chord sum over the
//                   near leaves (partials merged by TwoSum) + order-4
//                   expansion of the far cells, or the full direct sum for
//                   a marked block; writes FP64 w
//   k_ff_mlp        (mlp.cu) learned correction on tensor cores, adds to w
#include <algorithm>
#include <cmath>
#include <cstring>
#include <numeric>
#include <vector>

#include <cuda_runtime.h>

#include "farfield_dev.cuh"
#include "ffmath.cuh"
#include "nbody.cuh"

namespace lpm {

namespace {

__constant__ ff::CplxTable kCplx = ff::make_cplx_table();

__global__ void k_ff_sort_src(const double4_16a* __restrict__ src, const int* __restrict__ perm,
                              int64_t n, float4* __restrict__ ys) {
  const int64_t k = blockIdx.x * int64_t(blockDim.x) + threadIdx.x;
  if (k >= n) return;
  const double4_16a s = src[perm[k]];
  ys[k] = make_float4(float(s.x), float(s.y), float(s.z), float(s.w));
}

// Fixed-order block reduction of NV values held by each of 128 threads (the
// result in every thread).
template <int NV, class T>
__device__ void block_sum128(T* v, T* sh) {
  const int t = threadIdx.x, lane = t & 31, w = t >> 5;
#pragma unroll
  for (int i = 0; i < NV; ++i) {
    T x = v[i];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) x += __shfl_down_sync(0xffffffffu, x, o);
    if (lane == 0) sh[w * NV + i] = x;
  }
  __syncthreads();
  if (t < NV) sh[4 * NV + t] = ((sh[t] + sh[NV + t]) + (sh[2 * NV + t] + sh[3 * NV + t]));
  __syncthreads();
#pragma unroll
  for (int i = 0; i < NV; ++i) v[i] = sh[4 * NV + i];
  __syncthreads();
}

template <class T>
__device__ T block_max128(T x, T* sh) {
  const int t = threadIdx.x, lane = t & 31, w = t >> 5;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) x = max(x, __shfl_down_sync(0xffffffffu, x, o));
  if (lane == 0) sh[w] = x;
  __syncthreads();
  x = max(max(sh[0], sh[1]), max(sh[2], sh[3]));
  __syncthreads();
  return x;
}

// One CTA (128 threads) per cell.
__global__ void __launch_bounds__(128) k_ff_cells(const float4* __restrict__ ys,
                                                  const int4* __restrict__ cells, int ncells,
                                                  float theta, float rmax,
                                                  float* __restrict__ cd) {
  // FP32 throughout the per-point passes and reductions (the FP64 pipe is
  // 1/64 of FP32 on this part; the expansion is evaluated in FP32 anyway)
  __shared__ float sh[5 * 40];
  __shared__ float msh[35];
  const int cell = blockIdx.x;
  if (cell >= ncells) return;
  const int4 ci = cells[cell];
  const int s0 = ci.x, n = ci.y, t = threadIdx.x;
  // pass 1: centre, S, sum g
  float a[5] = {0.f, 0.f, 0.f, 0.f, 0.f};
  // (loads eight points ahead: the few largest cells are read by one CTA, which
  // waited a memory latency per point of a thread; the sums keep their order)
#pragma unroll 8
  for (int i = t; i < n; i += 128) {
    const float4 p = ys[s0 + i];
    a[0] += p.x;
    a[1] += p.y;
    a[2] += p.z;
    a[3] += fabsf(p.w);
    a[4] += p.w;
  }
  block_sum128<5>(a, sh);
  // centre and frame: one thread (FP64 is 1/64 of FP32 on this part), shared
  __shared__ float geo[16];
  __shared__ double cnorm;
  if (t == 0) {
    const double c[3] = {a[0] / n, a[1] / n, a[2] / n};
    const double cn = sqrt(c[0] * c[0] + c[1] * c[1] + c[2] * c[2]);
    double nn[3] = {1, 0, 0};
    if (cn > 0) nn[0] = c[0] / cn, nn[1] = c[1] / cn, nn[2] = c[2] / cn;
    const double r[3] = {fabs(nn[2]) < 0.9 ? 0.0 : 1.0, 0.0, fabs(nn[2]) < 0.9 ? 1.0 : 0.0};
    double e1[3] = {r[1] * nn[2] - r[2] * nn[1], r[2] * nn[0] - r[0] * nn[2], r[0] * nn[1] - r[1] * nn[0]};
    const double l = sqrt(e1[0] * e1[0] + e1[1] * e1[1] + e1[2] * e1[2]);
    e1[0] /= l, e1[1] /= l, e1[2] /= l;
    const double e2[3] = {nn[1] * e1[2] - nn[2] * e1[1], nn[2] * e1[0] - nn[0] * e1[2],
                          nn[0] * e1[1] - nn[1] * e1[0]};
    for (int k = 0; k < 3; ++k) {
      geo[k] = float(c[k]);
      geo[3 + k] = float(e1[k]);
      geo[6 + k] = float(e2[k]);
      geo[9 + k] = float(nn[k]);
    }
    cnorm = cn;
  }
  __syncthreads();
  const float cf[3] = {geo[0], geo[1], geo[2]};
  float qf[9];
  for (int k = 0; k < 9; ++k) qf[k] = geo[3 + k];
  const double cn = cnorm;
  // pass 2: radius about the (FP32) centre
  float hmax = 0.f;
#pragma unroll 8
  for (int i = t; i < n; i += 128) {
    const float4 p = ys[s0 + i];
    const float x0 = p.x - cf[0], x1 = p.y - cf[1], x2 = p.z - cf[2];
    hmax = fmaxf(hmax, x0 * x0 + x1 * x1 + x2 * x2);
  }
  const double h = sqrt(double(block_max128(hmax, sh)));
  // no target (all within rmax of the origin) can accept a cell whose radius
  // exceeds theta * (|c| + rmax): its moments are never used
  const bool skip = h > double(theta) * (cn + double(rmax));
  // pass 3: moments in the cell frame
  float m[35];
#pragma unroll
  for (int k = 0; k < 35; ++k) m[k] = 0.f;
  {
    for (int i = skip ? n : t; i < n; i += 128) {
      const float4 p = ys[s0 + i];
      const float x0 = p.x - cf[0], x1 = p.y - cf[1], x2 = p.z - cf[2];
      const float d0 = qf[0] * x0 + qf[1] * x1 + qf[2] * x2;
      const float d1 = qf[3] * x0 + qf[4] * x1 + qf[5] * x2;
      const float d2 = qf[6] * x0 + qf[7] * x1 + qf[8] * x2;
      float p0[5], p1[5], p2[5];
      p0[0] = p1[0] = p2[0] = 1.f;
#pragma unroll
      for (int k = 1; k <= 4; ++k) p0[k] = p0[k - 1] * d0, p1[k] = p1[k - 1] * d1, p2[k] = p2[k - 1] * d2;
      ff::sfor<35>([&](auto I) {
        constexpr int k = decltype(I)::value;
        m[k] = fmaf(p.w, p0[ff::mono_exp(k, 0)] * p1[ff::mono_exp(k, 1)] * p2[ff::mono_exp(k, 2)], m[k]);
      });
    }
  }
  block_sum128<35>(m, sh);
  if (t < 35) msh[t] = m[t];
  __syncthreads();
  const float* M = msh;
  // record: every thread holds the reduced moments; the fields are written
  // by different threads
  float* r = cd + int64_t(cell) * kCellF;
  if (t == 0) {
    r[0] = cf[0], r[1] = cf[1], r[2] = cf[2];
    r[3] = float(cn);
    r[4] = float(h);
    r[5] = float(a[3]);
    r[6] = float(a[4]);
    r[7] = float(n);
    for (int k = 0; k < 9; ++k) r[8 + k] = qf[k];
    for (int k = 63; k < kCellC; ++k) r[k] = 0.f;
    for (int k = kCellC + 35; k < kCellF; ++k) r[k] = 0.f;
  }
  if (t < 35) r[kCellM + t] = float(M[t]);
  if (t >= 35 && t < 45) {
    // traced moments sum g d^b |d|^2, |b| <= 2
    const int k = t - 35;
    double v = 0;
    ff::sfor<10>([&](auto I) {
      constexpr int i = decltype(I)::value;
      constexpr int e0 = ff::mono_exp(i, 0), e1 = ff::mono_exp(i, 1), e2 = ff::mono_exp(i, 2);
      if (i == k)
        v = M[ff::mono_index(e0 + 2, e1, e2)] + M[ff::mono_index(e0, e1 + 2, e2)] +
            M[ff::mono_index(e0, e1, e2 + 2)];
    });
    r[kCellN1 + k] = float(v);
  }
  if (t == 45) {
    // sum g |d|^4
    r[kCellN2] = float(M[ff::mono_index(4, 0, 0)] + M[ff::mono_index(0, 4, 0)] +
                       M[ff::mono_index(0, 0, 4)] +
                       2.0 * (M[ff::mono_index(2, 2, 0)] + M[ff::mono_index(2, 0, 2)] +
                              M[ff::mono_index(0, 2, 2)]));
  }
  if (t >= 64 && t < 64 + 35) {
    // complex moments normalised by S h^(p+q+k)
    const int j = t - 64;
    const double S = a[3] > 0 ? a[3] : 1.0;
    const double hh = h > 0 ? h : 1.0;
    double v = 0;
    for (int m = 0; m < kCplx.nterm[j]; ++m) v += double(kCplx.coef[j][m]) * M[kCplx.idx[j][m]];
    double nrm = S;
    for (int e = 0; e < kCplx.deg[j]; ++e) nrm *= hh;
    r[kCellC + j] = float(v / nrm);
  }
}

// One CTA (128 threads) per target block: Morton-ordered FP32 positions and
// the block's bounding sphere.
__global__ void __launch_bounds__(128) k_ff_tblocks(const double4_16a* __restrict__ tgt,
                                                    const int* __restrict__ tslot,
                                                    float4* __restrict__ xt, float4* __restrict__ box) {
  __shared__ double sh[5 * 8];
  __shared__ float fsh[4], ctr[3];
  const int64_t b = blockIdx.x;
  const int t = threadIdx.x;
  const int64_t i = b * kTargetBlock + t;
  float4 x = make_float4(0.f, 0.f, 0.f, 0.f);
  if (tslot[i] >= 0) {
    const double4_16a p = tgt[tslot[i]];
    x = make_float4(float(p.x), float(p.y), float(p.z), 1.f);
  }
  xt[i] = x;
  // FP64 sums (64 clocks a warp and operation): only of the coordinates, and
  // divided once per block
  const int count = __syncthreads_count(x.w > 0.f);
  double a[3] = {x.x, x.y, x.z};
  block_sum128<3>(a, sh);
  if (t < 3) ctr[t] = float((t == 0 ? a[0] : t == 1 ? a[1] : a[2]) / double(count));
  __syncthreads();
  const float c0 = ctr[0], c1 = ctr[1], c2 = ctr[2];
  float r = 0.f;
  if (x.w > 0) {
    const float e0 = x.x - c0, e1 = x.y - c1, e2 = x.z - c2;
    r = sqrtf(e0 * e0 + e1 * e1 + e2 * e2);
  }
  r = block_max128(r, fsh);
  if (t == 0) box[b] = make_float4(c0, c1, c2, r * (1.f + 1e-6f) + 1e-7f);
}

// The walk's verdict on a cell for one target block.
struct Verdict {
  bool far, learn, near;  // none: descend
};
__device__ __forceinline__ Verdict judge(const float* __restrict__ r, const int4 ci, const float4 bx,
                                         float theta, float rho_min, int learn) {
  const float e0 = bx.x - r[0], e1 = bx.y - r[1], e2 = bx.z - r[2];
  const float D = sqrtf(e0 * e0 + e1 * e1 + e2 * e2) - bx.w;
  const float h = r[4];
  const bool accept = D > 0.f && h <= theta * D;
  Verdict v;
  v.far = accept && ci.y >= kExactMax;
  v.learn = v.far && learn && h >= rho_min * D;
  // a leaf that is near, or far but small enough to sum exactly
  v.near = !v.far && ci.w == 0;
  return v;
}

// Depth-first walk from the root by one thread (a block whose list outgrows the
// warp's buffers).
__device__ __noinline__ int4 walk_serial(const float* __restrict__ cd, const int4* __restrict__ cells,
                                         float4 bx, float theta, float rho_min, int learn,
                                         int* __restrict__ F, int* __restrict__ N,
                                         int* __restrict__ L) {
  int stk[8 * 22];
  int sp = 0;
  stk[sp++] = 0;
  int nf = 0, nn = 0, nl = 0, over = 0;
  while (sp > 0) {
    const int c = stk[--sp];
    const int4 ci = cells[c];
    const Verdict v = judge(cd + int64_t(c) * kCellF, ci, bx, theta, rho_min, learn);
    if (v.far) {
      if (nf < kFarCap) F[nf] = c;
      nf++;
      if (v.learn) {
        if (nl < kLearnCap) L[nl] = c;
        nl++;
      }
    } else if (v.near) {
      if (nn < kNearCap) N[nn] = c;
      nn++;
    } else {
      if (sp + ci.w > 8 * 22) {
        over = 1;
        break;
      }
      for (int k = ci.w - 1; k >= 0; --k) stk[sp++] = ci.z + k;
    }
  }
  return make_int4(nf, nn, nl, over);
}

// One warp per target block.  The walk keeps an ordered list of cells and, level
// by level, judges 32 of them at a time: a far cell or a near leaf stays in place
// with a tag, any other is replaced by its children, so the list ends in the
// depth-first order of the serial walk.  A thread walking alone waited two memory
// latencies per cell: 253 us at icosahedral level 6, theta 0.4 (1,600 blocks),
// where the warp takes 22.
constexpr int kListCap = 2048;  // entries of the ordered list; beyond, walk_serial
constexpr int kListWarps = 2;
constexpr int kTagFar = 1 << 30, kTagNear = 1 << 29, kTagLearn = 1 << 28;  // cells < 2^28

__global__ void __launch_bounds__(32 * kListWarps) k_ff_lists(
    const float* __restrict__ cd, const int4* __restrict__ cells, const float4* __restrict__ box,
    int64_t nblocks, float theta, float rho_min, int learn, int* __restrict__ far,
    int* __restrict__ near, int* __restrict__ lrn, int4* __restrict__ cnt) {
  __shared__ int list[kListWarps][2][kListCap];
  const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const unsigned below = (1u << lane) - 1u;
  const int64_t b = blockIdx.x * int64_t(kListWarps) + w;
  if (b >= nblocks) return;
  const float4 bx = box[b];
  int* F = far + b * kFarCap;
  int* N = near + b * kNearCap;
  int* L = lrn + b * kLearnCap;
  int* in = list[w][0];
  int* out = list[w][1];
  if (lane == 0) in[0] = 0;
  __syncwarp();
  int len = 1;
  bool fits = true, open = true;
  while (open && fits) {
    open = false;
    int n = 0;
    for (int base = 0; base < len; base += 32) {
      int e = base + lane < len ? in[base + lane] : 0;
      int put = base + lane < len ? 1 : 0, child = -1;
      if (put && e < kTagLearn) {
        const int4 ci = cells[e];
        const Verdict v = judge(cd + int64_t(e) * kCellF, ci, bx, theta, rho_min, learn);
        if (v.far) {
          e |= kTagFar | (v.learn ? kTagLearn : 0);
        } else if (v.near) {
          e |= kTagNear;
        } else {
          child = ci.z;
          put = ci.w;
        }
      }
      open |= child >= 0;
      int x = put;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int y = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= o) x += y;
      }
      const int total = __shfl_sync(0xffffffffu, x, 31);
      if (n + total > kListCap) {
        fits = false;
        break;
      }
      const int at = n + x - put;
      if (child < 0) {
        if (put) out[at] = e;
      } else {
        for (int k = 0; k < put; ++k) out[at + k] = child + k;
      }
      n += total;
    }
    open = __any_sync(0xffffffffu, open);
    __syncwarp();
    int* s = in;
    in = out;
    out = s;
    len = n;
  }
  int4 c = make_int4(0, 0, 0, 0);
  if (fits) {
    for (int base = 0; base < len; base += 32) {
      const int e = base + lane < len ? in[base + lane] : 0;
      const int id = e & (kTagLearn - 1);
      const unsigned mf = __ballot_sync(0xffffffffu, (e & kTagFar) != 0);
      const unsigned mn = __ballot_sync(0xffffffffu, (e & kTagNear) != 0);
      const unsigned ml = __ballot_sync(0xffffffffu, (e & kTagLearn) != 0);
      int p = c.x + __popc(mf & below);
      if ((e & kTagFar) && p < kFarCap) F[p] = id;
      p = c.y + __popc(mn & below);
      if ((e & kTagNear) && p < kNearCap) N[p] = id;
      p = c.z + __popc(ml & below);
      if ((e & kTagLearn) && p < kLearnCap) L[p] = id;
      c.x += __popc(mf), c.y += __popc(mn), c.z += __popc(ml);
    }
  } else if (lane == 0) {
    c = walk_serial(cd, cells, bx, theta, rho_min, learn, F, N, L);
  }
  if (lane == 0) {
    const int over = c.w || c.x > kFarCap || c.y > kNearCap || c.z > kLearnCap;
    cnt[b] = make_int4(min(c.x, kFarCap), min(c.y, kNearCap), min(c.z, kLearnCap), over);
  }
}

constexpr int kNearBuf = 512;
constexpr int kFarBatch = 16;

__device__ __forceinline__ void chord_acc(float x0, float x1, float x2, float4 s, float c0,
                                          float& w0, float& w1, float& w2) {
  const float d0 = x0 - s.x, d1 = x1 - s.y, d2 = x2 - s.z;
  const float q = fmaf(d0, d0, fmaf(d1, d1, fmaf(d2, d2, c0)));
  const float r = s.w * rcp_approx(q);
  w0 = fmaf(r, d0, w0);
  w1 = fmaf(r, d1, w1);
  w2 = fmaf(r, d2, w2);
}

// One CTA (128 threads, one target each) per target block and part: part 0 sums
// the near leaves, and the far batches go to the parts in turn; the parts' FP64
// partials are added by the epilogue.  One part while the blocks fill the GPU for
// many waves, more where the last wave would leave it idle (ff_parts).
__global__ void __launch_bounds__(128) k_ff_eval(
    const float4* __restrict__ xt, const int* __restrict__ tslot,
    const float4* __restrict__ ys, int64_t nsrc, const float* __restrict__ cd,
    const int4* __restrict__ cells, const int* __restrict__ far, const int* __restrict__ near,
    const int4* __restrict__ cnt, float c0, double* __restrict__ wout, int64_t wstride) {
  __shared__ __align__(32) float4 buf[kNearBuf];  // read as 32-byte source pairs
  __shared__ float cell[kFarBatch][kCellF];
  __shared__ int4 lf[8];
  const int64_t b = blockIdx.x;
  const int t = threadIdx.x, part = blockIdx.y, parts = gridDim.y;
  const float4 x = xt[b * kTargetBlock + t];
  const int4 nc = cnt[b];
  float S0 = 0.f, S1 = 0.f, S2 = 0.f, C0 = 0.f, C1 = 0.f, C2 = 0.f;
  if (nc.w) {
    // lists overflowed: full direct sum (fallback), by part 0
    for (int64_t j0 = 0; j0 < (part == 0 ? nsrc : 0); j0 += kNearBuf) {
      const int m = int(nsrc - j0 < kNearBuf ? nsrc - j0 : kNearBuf);
      __syncthreads();
      for (int i = t; i < m; i += 128) buf[i] = ys[j0 + i];
      __syncthreads();
      float w0 = 0.f, w1 = 0.f, w2 = 0.f;
      for (int i = 0; i < m; ++i) chord_acc(x.x, x.y, x.z, buf[i], c0, w0, w1, w2);
      two_sum_acc(S0, C0, w0);
      two_sum_acc(S1, C1, w1);
      two_sum_acc(S2, C2, w2);
    }
  } else {
    // near leaves, up to 8 per batch (<= 512 sources); the 8 leaf records are
    // loaded by 8 threads at once
    const int* N = near + b * kNearCap;
    for (int l0 = 0; l0 < (part == 0 ? nc.y : 0); l0 += 8) {
      const int nl = min(8, nc.y - l0);
      __syncthreads();
      if (t < nl) lf[t] = cells[N[l0 + t]];
      __syncthreads();
      // sources staged as interleaved pairs (x0 x1 y0 y1 z0 z1 g0 g1) so that
      // one f32x2 instruction applies two sources to this thread's target
      float* pb = reinterpret_cast<float*>(buf);
      int o = 0;
      for (int k = 0; k < nl; ++k) {
        const int4 ci = lf[k];
        const int m = min(ci.y, kMaxLeaf);
        for (int i = t; i < m; i += 128) {
          const float4 v = ys[ci.x + i];
          float* e = pb + 8 * ((o + i) >> 1) + ((o + i) & 1);
          e[0] = v.x;
          e[2] = v.y;
          e[4] = v.z;
          e[6] = v.w;
        }
        o += m;
      }
      if ((o & 1) && t == 0) {  // odd count: a zero-strength partner at the origin
        float* e = pb + 8 * (o >> 1) + 1;
        e[0] = e[2] = e[4] = e[6] = 0.f;
      }
      __syncthreads();
      const u64 X2 = pk2(x.x, x.x), Y2 = pk2(x.y, x.y), Z2 = pk2(x.z, x.z), C02 = pk2(c0, c0);
      u64 W0 = 0ull, W1 = 0ull, W2 = 0ull;
      const ulonglong4_16a* pr = reinterpret_cast<const ulonglong4_16a*>(buf);
#pragma unroll 4
      for (int i = 0; i < (o + 1) >> 1; ++i) {
        const ulonglong4_16a s = pr[i];  // (x0 x1) (y0 y1) (z0 z1) (g0 g1)
        const u64 dx = sub2(X2, s.x), dy = sub2(Y2, s.y), dz = sub2(Z2, s.z);
        const u64 q = fma2(dx, dx, fma2(dy, dy, fma2(dz, dz, C02)));
        float qa, qb;
        upk2(q, qa, qb);
        const u64 w = mul2(s.w, pk2(rcp_approx(qa), rcp_approx(qb)));
        W0 = fma2(w, dx, W0);
        W1 = fma2(w, dy, W1);
        W2 = fma2(w, dz, W2);
      }
      float a0, b0, a1, b1, a2, b2;
      upk2(W0, a0, b0);
      upk2(W1, a1, b1);
      upk2(W2, a2, b2);
      two_sum_acc(S0, C0, a0 + b0);
      two_sum_acc(S1, C1, a1 + b1);
      two_sum_acc(S2, C2, a2 + b2);
      // leaves larger than kMaxLeaf (coincident points at the deepest level)
      for (int k = 0; k < nl; ++k) {
        const int4 ci = lf[k];
        if (ci.y <= kMaxLeaf) continue;
        float v0 = 0.f, v1 = 0.f, v2 = 0.f;
        for (int i = kMaxLeaf; i < ci.y; ++i) chord_acc(x.x, x.y, x.z, ys[ci.x + i], c0, v0, v1, v2);
        two_sum_acc(S0, C0, v0);
        two_sum_acc(S1, C1, v1);
        two_sum_acc(S2, C2, v2);
      }
    }
    // far cells: order-4 expansion, kFarBatch cells per batch
    const int* F = far + b * kFarCap;
    for (int f0 = part * kFarBatch; f0 < nc.x; f0 += parts * kFarBatch) {
      const int nb = min(kFarBatch, nc.x - f0);
      __syncthreads();
      for (int i = t; i < nb * kCellF; i += 128) {
        const int k = i / kCellF, e = i - k * kCellF;
        cell[k][e] = cd[int64_t(F[f0 + k]) * kCellF + e];
      }
      __syncthreads();
      float w0 = 0.f, w1 = 0.f, w2 = 0.f;
      for (int k = 0; k < nb; ++k) {
        float d[3], W[3], G[3];
        ff::to_cell(cell[k], x.x, x.y, x.z, d);
        ff::expand4(cell[k], d[0], d[1], d[2], c0, W);
        ff::from_cell(cell[k], W, G);
        w0 -= G[0];
        w1 -= G[1];
        w2 -= G[2];
      }
      two_sum_acc(S0, C0, w0);
      two_sum_acc(S1, C1, w1);
      two_sum_acc(S2, C2, w2);
    }
  }
  const int64_t tt = tslot[b * kTargetBlock + t];
  if (tt >= 0) {
    double* w = wout + 3 * part * wstride;
    w[tt] = double(S0) + double(C0);
    w[wstride + tt] = double(S1) + double(C1);
    w[2 * wstride + tt] = double(S2) + double(C2);
  }
}

}  // namespace

FFDevice::~FFDevice() {
  for (auto& c : caps) cudaFree(*c.first);
}
void FFDevice::reserve(void** p, size_t bytes) {
  if (*p) cudaFree(*p);  // waits for the device
  *p = nullptr;
  caps[p] = 0;
  LPM_CUDA(cudaMalloc(p, bytes));
}

void ff_cells(lpm_context& ctx, const float4* ys, const int4* cells, int ncells, float* cd) {
  k_ff_cells<<<ncells, 128, 0, ctx.stream>>>(ys, cells, ncells, 1.0f, 1e30f, cd);
  ctx.launches++;
  LPM_CUDA(cudaGetLastError());
}

// Parts of an evaluation: at least kPartWaves waves of seven CTAs per SM (six are
// resident, at 79 registers).  Icosahedral level 6, theta 0.4 (1,628 blocks: 1.8 waves in
// one part): 470 us in one part, 407 in three; level 8 (25,557 blocks) runs one part.
int ff_parts(const lpm_context& ctx, int64_t nblocks) {
  constexpr int64_t kPartWaves = 6;
  const int64_t slots = int64_t(std::max(ctx.num_sms, 1)) * 7;
  return int(std::max<int64_t>(1, std::min<int64_t>(kFFMaxParts, kPartWaves * slots / std::max<int64_t>(nblocks, 1))));
}

void ff_launch_tree(lpm_context& ctx, FFDevice& d, const void* tgt, const void* src, double* wout,
                    int64_t wstride, double c0, double theta, double rho_min, bool learn) {
  cudaStream_t st = ctx.stream;
  k_ff_sort_src<<<unsigned((d.nsrc + 255) / 256), 256, 0, st>>>(static_cast<const double4_16a*>(src),
                                                                 d.perm, d.nsrc, d.ys);
  k_ff_cells<<<d.ncells, 128, 0, st>>>(d.ys, d.cells, d.ncells, float(theta), d.rmax, d.cd);
  k_ff_tblocks<<<unsigned(d.nblocks), 128, 0, st>>>(static_cast<const double4_16a*>(tgt), d.tslot,
                                                    d.xt, d.box);
  k_ff_lists<<<unsigned((d.nblocks + kListWarps - 1) / kListWarps), 32 * kListWarps, 0, st>>>(
      d.cd, d.cells, d.box, d.nblocks, float(theta), float(rho_min), learn, d.far, d.near, d.lrn,
      d.cnt);
  k_ff_eval<<<dim3(unsigned(d.nblocks), unsigned(ff_parts(ctx, d.nblocks))), 128, 0, st>>>(d.xt, d.tslot, d.ys, d.nsrc, d.cd,
                                                 d.cells, d.far, d.near, d.cnt, float(c0), wout,
                                                 wstride);
  ctx.launches += 5;
  LPM_CUDA(cudaGetLastError());
}

}  // namespace lpm

// ---------------------------------------------------------------------------
// lpm_farfield host methods
// ---------------------------------------------------------------------------
lpm_farfield::~lpm_farfield() {
  for (void* e : events) cudaEventDestroy(static_cast<cudaEvent_t>(e));
  delete d;
}

int lpm_farfield::parts() const { return lpm::ff_parts(*ctx, d->nblocks); }

bool lpm_farfield::built() const { return d != nullptr && d->ncells > 0; }

void lpm_farfield::enter() {
  using namespace lpm;
  if (used && last_stream != ctx->stream) LPM_CUDA(cudaDeviceSynchronize());
  last_stream = ctx->stream;
  used = true;
}

void lpm_farfield::build(const double* src, int src_stride, int64_t nsrc, const double* tgt,
                         int tgt_stride, int64_t ntgt) {
  using namespace lpm;
  enter();
  ff_prepare_kernels();
  if (!d) d = new FFDevice();
  ++generation;
  d->ncells = 0;  // not built until the end
  build_tree_device(*ctx, *d, src, src_stride, nsrc, tgt, tgt_stride, ntgt, leaf_max);
}

void lpm_farfield::evaluate(const void* tgt, const void* src, double* wout, int64_t wstride,
                            double c0, double eps) {
  using namespace lpm;
  if (!built()) throw Error(LPM_ERR_STATE, "far field: tree not built");
  const bool learn = use_net && trained;
  cudaEvent_t ev[3] = {nullptr, nullptr, nullptr};
  if (timing) {
    for (auto& e : ev) {
      LPM_CUDA(cudaEventCreate(&e));
      events.push_back(e);
    }
    LPM_CUDA(cudaEventRecord(ev[0], ctx->stream));
  }
  ff_launch_tree(*ctx, *d, tgt, src, wout, wstride, c0, theta, rho_min, learn);
  if (timing) LPM_CUDA(cudaEventRecord(ev[1], ctx->stream));
  if (learn) ff_launch_mlp(*ctx, *d, *net, norm.data(), wout, wstride, eps, rho_min);
  if (timing) LPM_CUDA(cudaEventRecord(ev[2], ctx->stream));
}

void lpm_farfield::timings(double* tree_ms, double* net_ms, int64_t* evals) {
  using namespace lpm;
  LPM_CUDA(cudaStreamSynchronize(ctx->stream));
  double a = 0, b = 0;
  for (size_t i = 0; i + 2 < events.size(); i += 3) {
    float m0 = 0, m1 = 0;
    LPM_CUDA(cudaEventElapsedTime(&m0, static_cast<cudaEvent_t>(events[i]),
                                  static_cast<cudaEvent_t>(events[i + 1])));
    LPM_CUDA(cudaEventElapsedTime(&m1, static_cast<cudaEvent_t>(events[i + 1]),
                                  static_cast<cudaEvent_t>(events[i + 2])));
    a += m0;
    b += m1;
  }
  *tree_ms = a;
  *net_ms = b;
  *evals = int64_t(events.size() / 3);
  for (void* e : events) cudaEventDestroy(static_cast<cudaEvent_t>(e));
  events.clear();
}

void lpm_farfield::counts() {
  using namespace lpm;
  std::vector<int4> c(d->nblocks);
  LPM_CUDA(cudaMemcpyAsync(c.data(), d->cnt, sizeof(int4) * d->nblocks, cudaMemcpyDeviceToHost,
                           ctx->stream));
  LPM_CUDA(cudaStreamSynchronize(ctx->stream));
  last_far = last_near = last_learn = last_fallback = last_rows = 0;
  if (use_net && trained) {
    unsigned long long r = 0;
    LPM_CUDA(cudaMemcpy(&r, d->counter + 2, sizeof(r), cudaMemcpyDeviceToHost));
    last_rows = int64_t(r);
  }
  std::vector<int4> cells(d->ncells);
  LPM_CUDA(cudaMemcpy(cells.data(), d->cells, sizeof(int4) * d->ncells, cudaMemcpyDeviceToHost));
  std::vector<int> nearl(size_t(d->nblocks) * kNearCap);
  LPM_CUDA(cudaMemcpy(nearl.data(), d->near, sizeof(int) * nearl.size(), cudaMemcpyDeviceToHost));
  for (int64_t b = 0; b < d->nblocks; ++b) {
    if (c[b].w) {
      last_fallback++;
      continue;
    }
    last_far += c[b].x;
    last_learn += c[b].z;
    for (int k = 0; k < c[b].y; ++k) last_near += cells[nearl[b * kNearCap + k]].y;
  }
}
