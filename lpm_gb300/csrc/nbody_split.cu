// nbody_split.cu -- launches of the split FP64 sums (nbody_split.cuh): the
// range of the packed positions and strengths, the split source records, the
// pair kernel.
#include <algorithm>

#include "lpm_host.hpp"
#include "nbody_split.cuh"

namespace lpm {
namespace {

constexpr int kRangeThreads = 256;
constexpr int kSplitSums = 7;  // of k_split_pack's sources

// Magnitudes are compared by the high word of the double (exponent and 20
// mantissa bits): integer operations, where FP64 ones would take longer than
// the reads.  Values that are not finite do not count.
__device__ __forceinline__ int magnitude(double v) {
  const int h = __double2hiint(v) & 0x7fffffff;
  return h < 0x7ff00000 ? h : 0;
}
__device__ __forceinline__ bool not_finite(double v) {
  return (__double2hiint(v) & 0x7fffffff) >= 0x7ff00000;
}
__device__ __forceinline__ int exponent_above(int h) {  // values of magnitude h: < 2^result
  return (h >> 20) - 1022;
}

// Per-CTA largest magnitudes: source coordinates, strengths, target coordinates; and
// whether a source is not finite (an infinity has no float pair).
__global__ void __launch_bounds__(kRangeThreads)
    k_split_range(const double4_16a* __restrict__ tgt, int64_t nt,
                  const double4_16a* __restrict__ src, int64_t ns, int4* __restrict__ out,
                  SplitScale* __restrict__ scale) {
  __shared__ int sh[3];
  bool bad = false;
  if (threadIdx.x < 3) sh[threadIdx.x] = 0;
  if (blockIdx.x == 0 && threadIdx.x == 0) *scale = SplitScale{};
  __syncthreads();
  int ms = 0, mg = 0, mt = 0;
  const int64_t step = int64_t(gridDim.x) * kRangeThreads;
  const int64_t first = int64_t(blockIdx.x) * kRangeThreads + threadIdx.x;
#pragma unroll 4
  for (int64_t i = first; i < ns; i += step) {
    const double4_16a p = src[i];
    ms = max(ms, max(magnitude(p.x), max(magnitude(p.y), magnitude(p.z))));
    mg = max(mg, magnitude(p.w));
    bad |= not_finite(p.x) || not_finite(p.y) || not_finite(p.z) || not_finite(p.w);
  }
#pragma unroll 4
  for (int64_t i = first; i < nt; i += step) {
    const double4_16a p = tgt[i];
    mt = max(mt, max(magnitude(p.x), max(magnitude(p.y), magnitude(p.z))));
  }
  ms = __reduce_max_sync(0xffffffffu, ms);
  mg = __reduce_max_sync(0xffffffffu, mg);
  mt = __reduce_max_sync(0xffffffffu, mt);
  if ((threadIdx.x & 31) == 0) {
    atomicMax(&sh[0], ms);
    atomicMax(&sh[1], mg);
    atomicMax(&sh[2], mt);
  }
  const int any_bad = __syncthreads_or(bad);
  if (threadIdx.x == 0) out[blockIdx.x] = make_int4(sh[0], sh[1], sh[2], any_bad);
}

// Scales of the evaluation from the range kernel's partials (one warp).
__device__ SplitScale split_scale(const int4* __restrict__ part, int nparts, double eps) {
  int ms = 0, mg = 0, mt = 0;
  bool bad = false;
  for (int b = threadIdx.x; b < nparts; b += 32) {
    const int4 v = part[b];
    ms = max(ms, v.x), mg = max(mg, v.y), mt = max(mt, v.z);
    bad |= v.w != 0;
  }
  bad = __any_sync(0xffffffffu, bad);
  ms = __reduce_max_sync(0xffffffffu, ms);
  mg = __reduce_max_sync(0xffffffffu, mg);
  mt = __reduce_max_sync(0xffffffffu, mt);
  SplitScale s{};
  // targets up to eight times as far out as the sources are in range; others
  // (divided faces that ran away, say) take the FP64 path one by one
  const int es = exponent_above(ms), ep = exponent_above(magnitude(eps));
  const int ee = max(es, min(exponent_above(mt), es + 3));
  s.e = ms > 0 ? max(ee, ep) : 0;
  s.g = mg > 0 ? exponent_above(mg) : 0;
  if (bad || s.e < -400 || s.e > 400 || abs(s.g) > 400 || ep > (ms > 0 ? ee : 0) + 8) {
    s.big = 1;
    s.e = s.g = 0;
  }
  return s;
}

// The split records of the sources (pairs) and, in the blocks after them, of
// the targets; once per evaluation, so the pair kernel's CTAs (one per target
// block and chunk) start without FP64 work.  The sources' blocks also sum what the
// verdict goes by, in integers (in any order the same).
__global__ void __launch_bounds__(128)
    k_split_pack(const double4_16a* __restrict__ src, int64_t nsrc, int64_t npairs,
                 const double4_16a* __restrict__ tgt, int64_t ntgt, int64_t ntgt_pad, double eps,
                 const int4* __restrict__ part, int nparts, SplitPair* __restrict__ sp,
                 SplitTarget* __restrict__ st, SplitFixed* __restrict__ ps,
                 SplitFixed* __restrict__ pt, SplitScale* __restrict__ scale) {
  __shared__ SplitScale sc;
  if (threadIdx.x < 32) {
    const SplitScale s = split_scale(part, nparts, eps);
    if (threadIdx.x == 0) {
      sc = s;
      if (blockIdx.x == 0) scale->e = s.e, scale->g = s.g, scale->big = s.big;
    }
  }
  __syncthreads();
  const double xs = pow2d(-sc.e), gs = pow2d(-sc.g);
  const int64_t src_blocks = (npairs + 127) / 128;
  if (int64_t(blockIdx.x) >= src_blocks) {
    const int64_t i = (int64_t(blockIdx.x) - src_blocks) * 128 + threadIdx.x;
    if (i >= ntgt_pad) return;
    const double4_16a t = tgt[i];
    const double x = t.x * xs, y = t.y * xs, z = t.z * xs;
    SplitTarget r;
    r.x = split3(x), r.y = split3(y), r.z = split3(z);
    const double off = unit_defect(t.x, t.y, t.z);
    split2((2.0 * eps * eps + off) * xs * xs, r.ch, r.cl);
    r.exact = i < ntgt && (fabs(off) > 1.0 || fabs(x) >= 1.0 || fabs(y) >= 1.0 ||
                           fabs(z) >= 1.0);
    st[i] = r;
    if (pt) {
      // padding and positions that are NaN: any argument of the common path (the origin's
      // is next to 1, the logarithm's rare case); NaN is added to the sum
      const bool nan = isnan(t.x + t.y + t.z);
      pt[i] = i < ntgt && !nan
                  ? split_fixed(t, sc.e, off + 2.0 * eps * eps, 0.0, r.exact != 0)
                  : SplitFixed{0, 0, 0, 1ll << 61, nan ? t.x + t.y + t.z : 0.0, 0, 0};
    }
    return;
  }
  const int64_t k = int64_t(blockIdx.x) * 128 + threadIdx.x;
  // |g|, g^2, g, |g| y of the thread's sources in fixed point, and those off the sphere
  int sum[kSplitSums] = {};
  // padding: zero strength, outside the domain, so no denominator is zero
  float3 p[2][3];
  float2 gh, gl, ch, cl;
  int2 slot;
  auto put = [](float2& v, int j, float a) { (j == 0 ? v.x : v.y) = a; };
#pragma unroll
  for (int j = 0; j < 2; ++j) {
    const int64_t i = 2 * k + j;
    const bool real = i < nsrc;
    const double4_16a s = real ? src[i] : make_double4_16a(0, 0, 0, 0);
    p[j][0] = real ? split3(s.x * xs) : make_float3(4.f, 0.f, 0.f);
    p[j][1] = split3(s.y * xs);
    p[j][2] = split3(s.z * xs);
    float h, l;
    split2(-s.w * gs, h, l);
    put(gh, j, h), put(gl, j, l);
    const int f = __float2int_rn(-h * 0x1p20f);
    sum[0] += abs(f);
    sum[1] += __float2int_rn(h * h * 0x1p24f);
    sum[2] += f;
    sum[3] += __float2int_rn(fabsf(h) * 0x1p20f * p[j][0].x);
    sum[4] += __float2int_rn(fabsf(h) * 0x1p20f * p[j][1].x);
    sum[5] += __float2int_rn(fabsf(h) * 0x1p20f * p[j][2].x);
    const double off = real ? unit_defect(s.x, s.y, s.z) : 0.0;
    if (fabs(off) > 1.0) sum[6]++;
    // padding: a positive arg of no strength
    if (ps && k < npairs) ps[i] = real ? split_fixed(s, sc.e, off, s.w, false) : SplitFixed{0, 0, 0, 1ll << 61};
    split2(off * xs * xs, h, l);
    put(ch, j, h), put(cl, j, l);
    (j == 0 ? slot.x : slot.y) = real ? int(i) : -2;
  }
  SplitPair r;
  r.xh = make_float2(p[0][0].x, p[1][0].x);
  r.xm = make_float2(p[0][0].y, p[1][0].y);
  r.xl = make_float2(p[0][0].z, p[1][0].z);
  r.yh = make_float2(p[0][1].x, p[1][1].x);
  r.ym = make_float2(p[0][1].y, p[1][1].y);
  r.yl = make_float2(p[0][1].z, p[1][1].z);
  r.zh = make_float2(p[0][2].x, p[1][2].x);
  r.zm = make_float2(p[0][2].y, p[1][2].y);
  r.zl = make_float2(p[0][2].z, p[1][2].z);
  r.gh = gh, r.gl = gl, r.ch = ch, r.cl = cl;
  r.slot = slot;
  if (k < npairs) sp[k] = r;
  __shared__ int part_sum[4][kSplitSums];
#pragma unroll
  for (int q = 0; q < kSplitSums; ++q) {
    const int v = __reduce_add_sync(0xffffffffu, sum[q]);
    if ((threadIdx.x & 31) == 0) part_sum[threadIdx.x >> 5][q] = v;
  }
  __syncthreads();
  if (threadIdx.x < kSplitSums) {
    const int q = threadIdx.x;
    long long v = 0;
#pragma unroll
    for (int w = 0; w < 4; ++w) v += part_sum[w][q];
    atomicAdd(&scale->sum[q], (unsigned long long)(v));
  }
}

struct SplitBufs {
  int4* range;
  SplitScale* scale;
  SplitTarget* st;
  SplitPair* sp;
  SplitFixed *ps, *pt;  // nullptr: no stream function
};

template <bool SKIP>
void launch(lpm_context& ctx, const NbodyPlan& p, const SplitBufs& b, const double4_16a* tgt,
            const int* tself, const double4_16a* src, double* part, double eps) {
  const dim3 grid(unsigned(p.ntgt_pad / SPLIT_NT), unsigned(p.nchunks));
  if (p.wu) {
    nbody_split<SKIP><<<grid, SPLIT_NT, 0, ctx.stream>>>(
        tgt, tself, b.st, b.sp, src, b.scale, p.ntgt, p.ntgt_pad, p.nsrc, p.nsrc_pad, p.chunk_len,
        eps * eps, part, p.ncomp, ctx.d_err);
    ctx.launches++;
  }
  if (p.wp) {
    nbody_psi<SKIP><<<grid, SPLIT_NT, 0, ctx.stream>>>(tgt, tself, b.pt, b.ps, src, b.scale,
                                                       ctx.f64_tab, p.ntgt_pad, p.nsrc_pad,
                                                       p.chunk_len, eps * eps, part, p.ncomp);
    ctx.launches++;
  }
}

int range_blocks(const lpm_context& ctx, const NbodyPlan& p) {
  const int64_t want = (p.ntgt + p.nsrc + 4 * kRangeThreads - 1) / (4 * kRangeThreads);
  return int(std::max<int64_t>(1, std::min<int64_t>(want, 2 * std::max(ctx.num_sms, 1))));
}

size_t range_bytes(const lpm_context& ctx) {
  const size_t n = sizeof(int4) * size_t(2 * std::max(ctx.num_sms, 1));
  return (n + 255) / 256 * 256;
}

}  // namespace

size_t split_bytes(const lpm_context& ctx, int64_t ntgt_pad, int64_t nsrc_pad) {
  return 256 + range_bytes(ctx) + (sizeof(SplitTarget) + sizeof(SplitFixed)) * size_t(ntgt_pad) +
         (sizeof(SplitPair) / 2 + sizeof(SplitFixed)) * size_t(nsrc_pad);
}

void launch_split(lpm_context& ctx, const NbodyPlan& p, const void* tgt_, const int* tself,
                  const void* src_, double* part, double eps) {
  const auto* tgt = static_cast<const double4_16a*>(tgt_);
  const auto* src = static_cast<const double4_16a*>(src_);
  char* w = static_cast<char*>(p.split_buf);
  static_assert(sizeof(SplitScale) <= 256, "the scratch's first 256 bytes");
  SplitBufs b;
  b.scale = reinterpret_cast<SplitScale*>(w);
  b.range = reinterpret_cast<int4*>(w + 256);
  b.st = reinterpret_cast<SplitTarget*>(w + 256 + range_bytes(ctx));
  b.sp = reinterpret_cast<SplitPair*>(b.st + p.ntgt_pad);  // ntgt_pad is a multiple of 64
  b.ps = p.wp ? reinterpret_cast<SplitFixed*>(b.sp + p.nsrc_pad / 2) : nullptr;
  b.pt = p.wp ? b.ps + p.nsrc_pad : nullptr;
  const int nb = range_blocks(ctx, p);
  k_split_range<<<nb, kRangeThreads, 0, ctx.stream>>>(tgt, p.ntgt, src, p.nsrc, b.range, b.scale);
  const int64_t npairs = p.nsrc_pad / 2;
  k_split_pack<<<unsigned((npairs + 127) / 128 + (p.ntgt_pad + 127) / 128), 128, 0, ctx.stream>>>(
      src, p.nsrc, npairs, tgt, p.ntgt, p.ntgt_pad, eps, b.range, nb, b.sp, b.st, b.ps, b.pt, b.scale);
  ctx.launches += 2;
  if (p.skipc)
    launch<true>(ctx, p, b, tgt, tself, src, part, eps);
  else
    launch<false>(ctx, p, b, tgt, tself, src, part, eps);
}

}  // namespace lpm
