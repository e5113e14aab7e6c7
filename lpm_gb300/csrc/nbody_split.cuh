// nbody_split.cuh -- the FP64 sphere sums (LPM_FP64) on the FP32 pipe, by
// error-free transformations.
//
// Why: this part executes about 1.7 FP64 FMAs per clock per SM against 128
// FP32 ones, so the 8 FP64 operations of a pair (nbody_f64h) cost as much
// pipe time as 500 FP32 operations.  The form below takes about 160 FP32
// operations per sphere pair and keeps the accuracy of the FP64 kernels:
//
//  * Positions are scaled by a power of two into (-1, 1) and cut into three
//    floats on the common grids 2^-22 and 2^-45 (and the rest): differences of
//    like parts are exact, so d = x - y is exact before it is rounded to a
//    float pair (Dh, Dl) of 48 bits.  No cancellation error at all, where
//    1 - x.y in FP64 loses 1e-16 absolute.
//  * arg' = 2 (1 - x.y + eps^2) = |d|^2 + C as a float pair (exact products by
//    FMA, Knuth TwoSum), C = (1 - |x|^2) + (1 - |y|^2) + 2 eps^2; the defects
//    are taken exactly in FP64 once per point (they carry the reference's
//    behaviour at stage positions off the sphere).
//  * q = g / arg' as a float pair: MUFU reciprocal, one Newton step in FP32,
//    one residual; then q d as float pairs.
//  * Sums: float pairs over 4 steps, then three-float sums, then FP64 per chunk.
//  * The stream function in 64-bit fixed point (nbody_psi).
//
// A pair's term carries 5.2e-15 of random relative error (rms) and 1.3e-16 of
// mean error, which a sum of n like terms averages to 5.2e-15 sqrt(sum t^2) /
// |sum t|; the FP64 kernel's sum carries the rounding of the running sum and
// the cancellation in 1 - x.y (1e-16 / (1 - x.y) per pair, so the nearer a
// pair the more the split form is ahead: a target among the strong sources has
// errors of 1e-12 to 1e-14 in FP64, 1e-15 here).  For targets far from all strong
// sources FP64 is the better one where those are few (one: 7e-16 against 3e-15 of a
// velocity, 100: 3e-16 and 4e-16, 300 and 1,000: equal) or a compact cluster of
// both signs, whose sum t cancels (1e-15 against 5e-15).  So all pairs of an evaluation are
// in FP64 (split_verdict; the device decides, no launch depends on it) if the effective
// number of its sources, (sum |g|)^2 / sum g^2, is below a least one, or if their mean
// direction, weighted by |g|, is longer than 1/2 (strengths within about a hemisphere)
// and (sum g)^2 / sum g^2 is.  The least number: 256; and, as the velocity's error is
// 2e-14 (like signs: |sum g| of half sum |g| and more) to 6e-14 (a Rossby-Haurwitz wave)
// over its root and the FP64 form's is 2e-16 / max(mesh spacing, 2.7 eps), 100,000 eps^2
// for like signs, 500,000 eps^2 and 500,000 / sources for others (measured rms, split and
// FP64: wave, 1,280 sources, eps = 0.05 2.0e-15, 1.7e-15; 5,120 1.1e-15, 1.5e-15; eps =
// 0.2 1.2e-15, 0.6e-15; 81,920 0.74e-15, 0.76e-15).
// split_wanted() in direct_sum.cu holds the least sizes.
// Pairs closer than 2^-20 of the domain, where the float pairs would run out
// of bits, are evaluated in FP64 with the arithmetic of nbody_f64h.
//
// The planar and chord forms keep their FP64 kernels: they are well
// conditioned (3e-16 to 5e-16 against FP64 sums), and the same sums in this
// form measured 5e-16 to 1e-15.
//
// Off the sphere |d|^2 and C cancel, which leaves 2^-48 |C| of absolute error in
// arg'; up to |C| = 1/32 that is below the rounding of 1 - x.y itself.  Pairs
// with |C| above it and |arg'| < (|C| - 1/32) / 32 are evaluated in FP64 one by
// one (a run without reprojection drifts, and has stray points late on).
// Targets of |1 - |x|^2| > 1 or far outside the sources' range take the FP64
// path for all their pairs; all targets do when a sixteenth of the
// sources is that far off the sphere or eps is far larger than the domain.
// Measured on one GB300 (SM clock 2,070 MHz), pair kernel alone, velocity:
// icosahedral level 5 (10,242 x 20,480 pairs) 0.85 ms, 245 Gpairs/s, where 8 FP64
// operations per pair take 2.7 ms.  Bound: the FP32 pipe: 163 instructions, mostly
// f32x2 of two clocks each, per step of two sources fill 99 % of its clocks there.
#pragma once

#include "f32x2.cuh"
#include "nbody.cuh"

namespace lpm {

// Two sources, value by value: x hi, mid, lo (2 each), y, z, strength hi, lo,
// defect hi, lo, source indexes.
struct __align__(16) SplitPair {
  float2 xh, xm, xl, yh, ym, yl, zh, zm, zl, gh, gl, ch, cl;
  int2 slot;
};
static_assert(sizeof(SplitPair) == 112, "seven 16-byte loads per pair of sources");

constexpr int kSplitTile = SPLIT_TILE / 2;  // pairs of sources per tile
constexpr float kSplitTiny = 9.094947e-13f;  // 2^-40: a pair's least scaled arg'

// One point of the stream function: scaled position in units of 2^-61; its defect
// (targets: plus 2 eps^2) in units of 2^-58, with 32 bits after the point; a source's
// strength, or what is added to a target's sum (0 or NaN); whether a target lies
// outside the scaled range.
struct __align__(16) SplitFixed {
  long long x, y, z, c;
  double g;
  unsigned lo;
  int exact;
};

// One target: its three-float position, the constant part of arg' (its defect
// and 2 eps^2) and whether it lies outside the scaled range (the FP64 path).
struct __align__(16) SplitTarget {
  float3 x, y, z;
  float ch, cl;
  int exact;
};
static_assert(sizeof(SplitTarget) == 48, "three 16-byte loads per target");

// Scales of one evaluation, and what its verdict goes by: |position|, eps < 2^e,
// |strength| < 2^g.
struct SplitScale {
  int e, g;
  int big;  // out of range, not finite, or eps dwarfs the domain
  int pad;
  // of the sources' scaled strengths g in units of 2^-20 (g^2: 2^-24), two's complement
  unsigned long long sum[7];  // |g|, g^2, g, |g| y (3); sources of |1 - |y|^2| > 1
};

// Whether every pair is evaluated in FP64.
__device__ __forceinline__ bool split_verdict(const SplitScale& s, int64_t nsrc, double eps2) {
  auto v = [&](int q) { return float((long long)(s.sum[q])); };
  const float A = v(0), Q = 65536.f * v(1), G = v(2);  // Q in the others' units squared
  const float e2 = float(eps2);
  const float least =  // effective sources
      fmaxf(256.f, 4.f * G * G >= A * A ? 1e5f * e2 : 5e5f * fmaxf(1.f / float(nsrc), e2));
  const float k = s.big ? 0.f : exp2f(float(s.e));
  const float m0 = k * v(3), m1 = k * v(4), m2 = k * v(5);
  const bool compact = m0 * m0 + m1 * m1 + m2 * m2 > 0.25f * A * A;
  return s.big || s.sum[6] * 16 > (unsigned long long)(nsrc) || A * A < least * Q ||
         (compact && G * G < least * Q);
}

// 2^k for |k| <= 1022
__device__ __forceinline__ double pow2d(int k) {
  return __longlong_as_double((long long)(1023 + k) << 52);
}

// X in (-1, 1): x a multiple of 2^-22, y a multiple of 2^-45 with |y| <= 2^-23.
__device__ __forceinline__ float3 split3(double X) {
  const double m1 = 1.5 * 1073741824.0;                    // ulp 2^-22
  const double m2 = 1.5 * 128.0;                           // ulp 2^-45
  const double h = __dsub_rn(__dadd_rn(X, m1), m1);
  const double r = __dsub_rn(X, h);
  const double m = __dsub_rn(__dadd_rn(r, m2), m2);
  return make_float3(float(h), float(m), float(__dsub_rn(r, m)));
}
__device__ __forceinline__ void split2(double v, float& h, float& l) {
  h = float(v);
  l = float(v - double(h));
}
// 1 - |x|^2 to about 1e-31 absolute, rounded to FP64.
__device__ __forceinline__ double unit_defect(double x, double y, double z) {
  double s = 1.0, e = 0.0;
  const double v[3] = {x, y, z};
#pragma unroll
  for (int c = 0; c < 3; ++c) {
    const double p = __dmul_rn(v[c], v[c]);
    const double pe = fma(v[c], v[c], -p);
    const double t = __dsub_rn(s, p);
    const double bb = __dsub_rn(t, s);
    e += __dsub_rn(__dsub_rn(s, __dsub_rn(t, bb)), __dadd_rn(p, bb)) - pe;
    s = t;
  }
  return s + e;
}

__device__ __forceinline__ SplitFixed split_fixed(const double4_16a& p, int e, double off, double g,
                                                  bool exact) {
  const double k = pow2d(61 - e), c = off * pow2d(58 - 2 * e), f = floor(c);
  return SplitFixed{__double2ll_rn(p.x * k), __double2ll_rn(p.y * k), __double2ll_rn(p.z * k),
                    (long long)(f), g, unsigned((c - f) * 0x1p32), exact};
}

__device__ __forceinline__ void two_sum2(u64 a, u64 b, u64& s, u64& e) {
  s = add2(a, b);
  const u64 bb = sub2(s, a);
  e = add2(sub2(a, sub2(s, bb)), sub2(b, bb));
}
__device__ __forceinline__ void two_sum1(float a, float b, float& s, float& e) {
  s = a + b;
  const float bb = s - a;
  e = (a - (s - bb)) + (b - bb);
}
__device__ __forceinline__ u64 dup2(float a) { return pk2(a, a); }
__device__ __forceinline__ u64 pkf2(float2 a) { return pk2(a.x, a.y); }

// Running sum of float pairs: the two lanes' pairs are added first, then a
// float-pair sum over kSplitRun steps (16 FP32 operations per step), which is
// merged into a three-float sum.  The rounding of the low words grows with the
// run's partial sum, so the run is short: 4 steps leave it below the terms' own
// error (16 steps, or an unbroken three-float sum, left several times it).
constexpr int kSplitRun = 4;
struct SplitAcc {
  float s = 0.f, c = 0.f;
  float t0 = 0.f, t1 = 0.f, t2 = 0.f;
  __device__ __forceinline__ void add(u64 h, u64 l) {
    float h0, h1, l0, l1, e;
    upk2(h, h0, h1);
    upk2(l, l0, l1);
    two_sum1(h0, h1, h0, e);
    l0 = (l0 + l1) + e;
    two_sum1(s, h0, s, e);
    c += l0 + e;
  }
  __device__ __forceinline__ void merge() {
    float e, f;
    two_sum1(t0, s, t0, e);
    two_sum1(e, c, e, f);
    t2 += f;
    two_sum1(t1, e, t1, f);
    t2 += f;
    s = c = 0.f;
  }
  __device__ __forceinline__ double value() const { return double(t0) + (double(t1) + double(t2)); }
};

// One pair in FP64, the arithmetic of nbody_f64h, added to its partials.
__device__ __forceinline__ void split_pair64(const double4_16a& t, const double4_16a& s,
                                             double eps2, double* a) {
  const double arg = eps2 - fma(t.z, s.z, fma(t.y, s.y, fma(t.x, s.x, -1.0)));
  const double q = div_nr(s.w, arg);
  a[0] = fma(q, s.x, a[0]);
  a[1] = fma(q, s.y, a[1]);
  a[2] = fma(q, s.z, a[2]);
}
// The rare pair, out of line.
static __device__ __noinline__ void split_near64(const double4_16a* t, const double4_16a* s,
                                                 double eps2, double* a) {
  split_pair64(*t, *s, eps2, a);
}

// All pairs of one target and chunk with the operations of nbody_f64h, whose rate it
// has (the FP64 pipe bounds it; the sources are uniform loads), summed in runs of a tile:
// a split chunk may be several times as long as one of nbody_f64h.  Out of line, called
// before the split sums hold registers.
template <bool SKIP>
__device__ __noinline__ void split_fp64(const double4_16a* __restrict__ tgt,
                                        const int* __restrict__ tself,
                                        const double4_16a* __restrict__ src, int64_t ti, int64_t j0,
                                        int64_t j1, double eps2, double* __restrict__ out,
                                        int64_t ntgt_pad) {
  const double4_16a t = tgt[ti];
  const int self = SKIP ? tself[ti] : -1;
  double sum[3] = {0.0, 0.0, 0.0};
  for (int64_t i = j0; i < j1; i += SPLIT_TILE) {
    const int64_t end = i + SPLIT_TILE < j1 ? i + SPLIT_TILE : j1;
    double a[3] = {0.0, 0.0, 0.0};
#pragma unroll 2
    for (int64_t j = i; j < end; ++j) {
      const double4_16a s = src[j];
      const double arg = eps2 - fma(t.z, s.z, fma(t.y, s.y, fma(t.x, s.x, -1.0)));
      const double q = f64_plain(fabs(arg)) ? s.w * f64_rcp(arg) : div_nr_any(s.w, arg);
      const double g = SKIP && j == self ? 0.0 : q;
      a[0] = fma(g, s.x, a[0]);
      a[1] = fma(g, s.y, a[1]);
      a[2] = fma(g, s.z, a[2]);
    }
#pragma unroll
    for (int k = 0; k < 3; ++k) sum[k] += a[k];
  }
#pragma unroll
  for (int k = 0; k < 3; ++k) out[k * ntgt_pad + ti] = sum[k];
}

// ---- the stream function --------------------------------------------------------
// |d|^2 in units of 2^-58 (to about one).  The squares from 32-bit halves, D = h 2^32 + l
// with signed h and l: h^2 + 2 h l / 2^32, without l^2.
__device__ __forceinline__ long long split_square(const long long (&d)[3]) {
  long long T = 0, c = 0;
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    const int l = int(unsigned(d[k])), h = int(d[k] >> 32) + (l < 0);
    T += (long long)(h) * h;
    c += (long long)(h) * l;
  }
  return T + (c >> 31);
}
// arg = T 2^(e2 - 59) as a double, T > 0.
__device__ __forceinline__ double split_arg_value(long long T, int e2) {
  const int z = __clzll(T);
  return __longlong_as_double(int64_t(f64_pack(uint64_t(T) << z, 1023 + 63 - z + e2 - 59)));
}
// Sums below this (arg < 1e-6 on the unit sphere) keep too few bits; above, arg' is good
// to about 1.4e-17, where 1 - x.y in FP64 has 1e-16.
constexpr long long kPsiClose = 1ll << 37;
// arg in FP64: with ref (what the fixed point does not hold) as nbody_f64h, else from
// |d|^2, for pairs within about 1e-6.
static __device__ __noinline__ double split_arg64(const double4_16a* t, const double4_16a* s,
                                                  double eps2, bool ref) {
  if (ref) return eps2 - fma(t->z, s->z, fma(t->y, s->y, fma(t->x, s->x, -1.0)));
  const double d0 = t->x - s->x, d1 = t->y - s->y, d2 = t->z - s->z;
  const double c = unit_defect(t->x, t->y, t->z) + unit_defect(s->x, s->y, s->z) + 2.0 * eps2;
  return 0.5 * (fma(d0, d0, fma(d1, d1, d2 * d2)) + c);
}
// Any pair's arg.  A close one's d is taken k bits up, C from its bits after the point.
static __device__ __noinline__ double split_arg_any(long long d0, long long d1, long long d2,
                                                    long long C, unsigned lo, int e,
                                                    const double4_16a* t, const double4_16a* s,
                                                    double eps2, bool ref) {
  if (!ref) {
    long long d[3] = {d0, d1, d2};
    const long long m = llabs(d0) | llabs(d1) | llabs(d2);
    const int k = max(0, min(min(__clzll(m) - 2, (__clzll(llabs(C) | 1) - 3) / 2), 16));
#pragma unroll
    for (int q = 0; q < 3; ++q) d[q] *= 1ll << k;
    const long long T = split_square(d) + C * (1ll << (2 * k)) + (long long)(((unsigned long long)(lo) << (2 * k)) >> 32);
    if (T >= kPsiClose) return split_arg_value(T, 2 * (e - k));
  }
  return split_arg64(t, s, eps2, ref);
}

// Partials of the stream function, sum g log(arg): a logarithm carries arg's relative
// error as an absolute one, and far pairs weigh as much as near ones, so float pairs
// (5e-15 a pair) were 1.5 to 4 times further off than nbody_f64h on meshes of 1,280 to
// 6,144 sources.  Here arg is exact to 53 bits (no cancellation of 1 - x.y), formed in
// integers as its logarithm is (f64math.cuh): 3 FP64 operations per pair.  A kernel of
// its own: beside the float-pair velocity its registers left 16 warps per SM, which do
// not hide its chains of operations (velocity and stream function, 14,336 targets by
// 6,144 sources: 1.35 ms in one kernel, 1.08 ms in two, 2.46 ms as nbody_f64h, 0.75 ms
// in float pairs).  Bound: the FP64 pipe, 0.82 of its rate.
//   pt, ps: SplitFixed per target and source, ntgt_pad and nsrc_pad of them
//   part: [chunk][nc][ntgt_pad], the last component
template <bool SKIP>
__global__ void __launch_bounds__(SPLIT_NT, 16)
    nbody_psi(const double4_16a* __restrict__ tgt, const int* __restrict__ tself,
              const SplitFixed* __restrict__ pt, const SplitFixed* __restrict__ ps,
              const double4_16a* __restrict__ src, const SplitScale* __restrict__ scale,
              const F64Tables* __restrict__ tab, int64_t ntgt_pad, int64_t nsrc_pad, int chunk_len,
              double eps2, double* __restrict__ part, int nc) {
  const int64_t ti = (int64_t)blockIdx.x * SPLIT_NT + threadIdx.x;
  const int64_t s0 = (int64_t)blockIdx.y * chunk_len;
  const int64_t s1 = s0 + chunk_len < nsrc_pad ? s0 + chunk_len : nsrc_pad;
  const int e = scale->e;
  const SplitFixed x = pt[ti];
  const bool ref = scale->big != 0 || x.exact != 0;
  const int self = SKIP ? tself[ti] : -1;
  double sum = 0.0;
  for (int64_t i0 = s0; i0 < s1; i0 += SPLIT_TILE) {
    double run = 0.0;
#pragma unroll 1
    for (int64_t i = i0; i < i0 + SPLIT_TILE; i += 2) {
      // (two sources' chains side by side)
      const SplitFixed y0 = ps[i], y1 = ps[i + 1];
      const long long d0[3] = {x.x - y0.x, x.y - y0.y, x.z - y0.z};
      const long long d1[3] = {x.x - y1.x, x.y - y1.y, x.z - y1.z};
      // (a target's own source: any argument of the common path, left out below)
      const bool own0 = SKIP && i == self, own1 = SKIP && i + 1 == self;
      const long long T0 = own0 ? 1ll << 58 : split_square(d0) + (x.c + y0.c);
      const long long T1 = own1 ? 1ll << 58 : split_square(d1) + (x.c + y1.c);
      double a0 = split_arg_value(T0, 2 * e), a1 = split_arg_value(T1, 2 * e);
      if (ref || T0 < kPsiClose || T1 < kPsiClose) {
        const unsigned l0 = x.lo + y0.lo, l1 = x.lo + y1.lo;
        if (!own0)
          a0 = split_arg_any(d0[0], d0[1], d0[2], x.c + y0.c + (l0 < x.lo), l0, e, tgt + ti, src + i,
                             eps2, ref);
        if (!own1)
          a1 = split_arg_any(d1[0], d1[1], d1[2], x.c + y1.c + (l1 < x.lo), l1, e, tgt + ti,
                             src + i + 1, eps2, ref);
      }
      double v0, v1;
      if (f64_log_plain(a0) && f64_log_plain(a1)) {
        v0 = f64_log(tab, a0), v1 = f64_log(tab, a1);
      } else {
        v0 = f64_ln_any(a0), v1 = f64_ln_any(a1);
      }
      if (!own0) run = fma(v0, y0.g, run);
      if (!own1) run = fma(v1, y1.g, run);
    }
    sum += run;
  }
  part[((int64_t)blockIdx.y * nc + nc - 1) * ntgt_pad + ti] = sum + x.g;
}

// ---- the velocity ---------------------------------------------------------------
//   tgt, tself, src, part: as nbody_f64h (sphere forms)
//   st: SplitTarget per target (ntgt_pad entries)
//   sp: SplitPair per two sources (nsrc_pad / 2 entries)
//   SKIP: the pair of tself is left out
//   nc: components of the partials, the velocity's first
template <bool SKIP>
__global__ void __launch_bounds__(SPLIT_NT, 512 / SPLIT_NT)
    nbody_split(const double4_16a* __restrict__ tgt, const int* __restrict__ tself,
                const SplitTarget* __restrict__ st, const SplitPair* __restrict__ sp,
                const double4_16a* __restrict__ src, const SplitScale* __restrict__ scale,
                int64_t ntgt, int64_t ntgt_pad, int64_t nsrc, int64_t nsrc_pad, int chunk_len,
                double eps2, double* __restrict__ part, int nc, int* err) {
  constexpr int NC = 3;
  __shared__ __align__(128) SplitPair sbuf[2 * kSplitTile];
  __shared__ __align__(8) uint64_t sbar[2];
  const SplitScale sc = *scale;

  const int64_t ti = (int64_t)blockIdx.x * SPLIT_NT + threadIdx.x;
  const int64_t s0 = (int64_t)blockIdx.y * chunk_len;
  int64_t slen = nsrc_pad - s0;
  if (slen > chunk_len) slen = chunk_len;
  if (split_verdict(sc, nsrc, eps2)) {
    split_fp64<SKIP>(tgt, tself, src, ti, s0, s0 + slen < nsrc ? s0 + slen : nsrc, eps2,
                     part + (int64_t)blockIdx.y * nc * ntgt_pad, ntgt_pad);
    return;
  }
  TilePipe<SplitPair, kSplitTile> pipe{sbuf, sbar, sp + s0 / 2, int(slen / (2 * kSplitTile))};
  pipe.start();

  const SplitTarget t = st[ti];
  const int self = SKIP ? tself[ti] : -1;
  const bool exact = t.exact != 0;
  const u64 XH = dup2(t.x.x), XM = dup2(t.x.y), XL = dup2(t.x.z);
  const u64 YH = dup2(t.y.x), YM = dup2(t.y.y), YL = dup2(t.y.z);
  const u64 ZH = dup2(t.z.x), ZM = dup2(t.z.y), ZL = dup2(t.z.z);
  const u64 CH = dup2(t.ch), CL = dup2(t.cl);
  SplitAcc acc[3];
  double near[NC];  // what is evaluated in FP64, in the partials' units
#pragma unroll
  for (int k = 0; k < NC; ++k) near[k] = 0.0;
  // -1/1024 in the scale of arg'; padding targets take out nothing
  const float tiny = ti < ntgt ? kSplitTiny : -1e30f;
  const float off = ti < ntgt ? -float(pow2d(-2 * sc.e) / 1024) : -1e30f;
  const u64 one = dup2(1.f);

  // (a warp whose targets all do, or are padding, still passes its tiles, without
  // the sums)
  const bool idle = __all_sync(0xffffffffu, exact || ti >= ntgt);
  for (int tl = 0; tl < pipe.ntiles; ++tl) {
    if (!pipe.acquire(tl)) {
      pipe.drain(tl, err);
      return;
    }
    const SplitPair* sm = pipe.tile(tl);
#pragma unroll 1
    for (int j0 = 0; j0 < kSplitTile && !idle; j0 += kSplitRun) {
#pragma unroll 1
      for (int j = j0; j < j0 + kSplitRun; ++j) {
        const SplitPair s = sm[j];
        // exact differences, then a float pair
        u64 dh[3], dl[3], u, v;
        u = sub2(XH, pkf2(s.xh)), v = sub2(XM, pkf2(s.xm));
        dh[0] = add2(u, v);
        dl[0] = add2(sub2(v, sub2(dh[0], u)), sub2(XL, pkf2(s.xl)));
        u = sub2(YH, pkf2(s.yh)), v = sub2(YM, pkf2(s.ym));
        dh[1] = add2(u, v);
        dl[1] = add2(sub2(v, sub2(dh[1], u)), sub2(YL, pkf2(s.yl)));
        u = sub2(ZH, pkf2(s.zh)), v = sub2(ZM, pkf2(s.zm));
        dh[2] = add2(u, v);
        dl[2] = add2(sub2(v, sub2(dh[2], u)), sub2(ZL, pkf2(s.zl)));
        // |d|^2.  The low words' order matters for the mean error: the residual of
        // a square has patterned last bits (k^2 mod 4 is 0 or 1) that round down
        // when summed, so it enters under a product (2 dh dl) that rounds at
        // random; so do the tiny dl^2, which added to a word would always round
        // away.  As plain sums the two left 1e-15 of bias, which no averaging
        // over sources removes.
        const u64 p0 = mul2(dh[0], dh[0]), p1 = mul2(dh[1], dh[1]), p2 = mul2(dh[2], dh[2]);
        const u64 sq = fma2(dl[2], dl[2], fma2(dl[0], dl[0], mul2(dl[1], dl[1])));
        u64 lo = fma2(add2(dh[1], dh[1]), dl[1], sq);
        lo = add2(lo, fma2(dh[1], dh[1], neg2(p1)));
        lo = add2(lo, fma2(add2(dh[0], dh[0]), dl[0], fma2(dh[0], dh[0], neg2(p0))));
        u64 q, e;
        two_sum2(p0, p1, q, e);
        lo = add2(lo, e);
        lo = add2(lo, fma2(add2(dh[2], dh[2]), dl[2], fma2(dh[2], dh[2], neg2(p2))));
        two_sum2(q, p2, q, e);
        lo = add2(lo, e);
        // arg' = |d|^2 + C
        u64 c, A;
        two_sum2(CH, pkf2(s.ch), c, e);
        const u64 cl = add2(add2(CL, pkf2(s.cl)), e);
        two_sum2(q, c, A, e);
        u64 Al = add2(lo, add2(e, cl));
        float a0, a1;
        upk2(A, a0, a1);
        // pairs taken out (rare): the closest and those off the sphere,
        // evaluated in FP64, and the target's own source
        float c0, c1;
        upk2(c, c0, c1);
        const bool n0 = fabsf(a0) < fmaxf(tiny, fmaf(fabsf(c0), 1.f / 32, off)) ||
                        (SKIP && s.slot.x == self);
        const bool n1 = fabsf(a1) < fmaxf(tiny, fmaf(fabsf(c1), 1.f / 32, off)) ||
                        (SKIP && s.slot.y == self);
        u64 gh = pkf2(s.gh), gl = pkf2(s.gl);
        if (n0 || n1) {
          if (n0 && s.slot.x >= 0 && !(SKIP && s.slot.x == self))
            split_near64(tgt + ti, src + s.slot.x, eps2, near);
          if (n1 && s.slot.y >= 0 && !(SKIP && s.slot.y == self))
            split_near64(tgt + ti, src + s.slot.y, eps2, near);
          // strength 0 and denominator 1 in the split sum
          float b0, b1;
          upk2(Al, b0, b1);
          a0 = n0 ? 1.f : a0;
          a1 = n1 ? 1.f : a1;
          A = pk2(a0, a1);
          Al = pk2(n0 ? 0.f : b0, n1 ? 0.f : b1);
          gh = pk2(n0 ? 0.f : s.gh.x, n1 ? 0.f : s.gh.y);
          gl = pk2(n0 ? 0.f : s.gl.x, n1 ? 0.f : s.gl.y);
        }
        // r = -1 / arg': the MUFU's value, one Newton step, its residual
        u64 r = pk2(rcp_approx(-a0), rcp_approx(-a1));
        r = fma2(r, fma2(A, r, one), r);
        e = fma2(Al, r, fma2(A, r, one));
        const u64 rl = mul2(r, fma2(e, e, e));
        // the record holds -g: q = g / arg'
        const u64 qh = mul2(gh, r);
        u64 ql = fma2(gh, r, neg2(qh));
        ql = fma2(gh, rl, ql);
        ql = fma2(gl, r, ql);
#pragma unroll
        for (int k = 0; k < 3; ++k) {
          const u64 ph = mul2(qh, dh[k]);
          u64 pl = fma2(qh, dh[k], neg2(ph));
          pl = fma2(ql, dl[k], fma2(qh, dl[k], pl));
          pl = fma2(ql, dh[k], pl);
          acc[k].add(ph, pl);
        }
      }
#pragma unroll
      for (int c = 0; c < 3; ++c) acc[c].merge();
    }
    pipe.release(tl);
  }

  double* out = part + (int64_t)blockIdx.y * nc * ntgt_pad;
  const unsigned lanes = __ballot_sync(0xffffffffu, exact);
  if (lanes != 0) {
    // FP64 targets: each by its own thread where they fill half the warp, one
    // after another by the whole warp where they are few (a lone thread would
    // hold its warp for 40 times as long)
    const int64_t j1 = s0 + slen < nsrc ? s0 + slen : nsrc;
    const int lane = threadIdx.x & 31;
    const bool own = __popc(lanes) >= 16;
    for (unsigned rest = own ? 1u : lanes; rest != 0; rest &= rest - 1) {
      const int b = own ? lane : __ffs(rest) - 1;
      const int sb = __shfl_sync(0xffffffffu, self, b);
      const double4_16a x = tgt[ti - lane + b];
      double a[NC];
#pragma unroll
      for (int k = 0; k < NC; ++k) a[k] = 0.0;
      if (!own || exact) {
#pragma unroll 2
        for (int64_t j = s0 + (own ? 0 : lane); j < j1; j += own ? 1 : 32) {
          const double4_16a y = src[j];
          if (!(SKIP && j == sb)) split_pair64(x, y, eps2, a);
        }
      }
      if (!own) {
#pragma unroll
        for (int k = 0; k < NC; ++k)
#pragma unroll
          for (int o = 16; o > 0; o >>= 1) a[k] += __shfl_xor_sync(0xffffffffu, a[k], o);
      }
      if (lane == b && exact)
#pragma unroll
        for (int k = 0; k < NC; ++k) out[k * ntgt_pad + ti] = a[k];
    }
  }
  if (!exact) {
    // the sum of g d / arg' in the caller's units; -2 times it equals the sum
    // of (g / arg) y in the cross product with x
    const double f = -2.0 * pow2d(sc.g - sc.e);
#pragma unroll
    for (int k = 0; k < 3; ++k) near[k] += acc[k].value() * f;
#pragma unroll
    for (int k = 0; k < NC; ++k) out[k * ntgt_pad + ti] = near[k];
  }
}

}  // namespace lpm
