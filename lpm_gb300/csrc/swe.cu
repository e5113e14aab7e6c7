// swe.cu -- shallow-water direct sums: planar with particle strength exchange
// (PlanarSWEVertexSums / PlanarSWEFaceSums, src/lpm_swe_kernels.hpp:626-876)
// and spherical (SphereVertexSums / SphereFaceSums, :723-940; see
// k_swe_sphere below).
//
// Pair term (planar_swe_sums_rhs_pse, :394-480): with d = x - y,
// R = |d|^2 + eps^2, rot = zeta A, pot = sigma A,
//   u, v         = (-d1 rot + d0 pot) / (2 pi R), (d0 rot + d1 pot) / (2 pi R)
//   du/dx, du/dy, dv/dx, dv/dy from pi R^2 and 2 pi R denominators,
//   lap(s)       = (s_y - s_x) A lapPSE(|y - x| / pse_eps) / pse_eps^2,
//                  lapPSE(r) = (40 (1 - r^2) + 10 r^4 - 2 r^6 / 3) e^{-r^2} / pi
//                  (pse::BivariateOrder8::laplacian, src/lpm_pse.hpp:66-72),
//   psi, phi     = -log(R) / (4 pi) times rot, pot.
// Reducer rules (:559-570): masked sources are skipped; with collocated
// targets (face sums with eps = 0) the i == j pair is skipped.
//
// FP64 sums the pair terms as moments of d (k_swe_plane below); FP64 partials
// per (chunk, component, target) are added in fixed order by the epilogue,
// which assembles the outputs and the double dot product du/dx^2 +
// 2 du/dy dv/dx + dv/dy^2.
#include <algorithm>
#include <cmath>

#include <cuda_runtime.h>

#include "f64math.cuh"
#include "lpm_host.hpp"
#include "nbody.cuh"

namespace lpm {
int fail(int code, const char* msg);  // capi.cu
int handle_exception();               // capi.cu

namespace {

__device__ __forceinline__ double dm(double a, double b) { return __dmul_rn(a, b); }
__device__ __forceinline__ double da(double a, double b) { return __dadd_rn(a, b); }
__device__ __forceinline__ double ds(double a, double b) { return __dsub_rn(a, b); }

constexpr int kSweNT = 128;   // targets per CTA
constexpr int kSweTile = 256;  // sources per shared-memory tile (FP32)
// FP64: small tiles and chunks, so that a few thousand points spread evenly
// (a warp's pair takes 1,200 to 3,000 clocks of its sub-partition's FP64 pipe)
constexpr int kSweTile64 = 64;

// ---- planar SWE sums, FP64 --------------------------------------------------
// With e = d / R, the eleven sums
//   U, V    = sum -rot e1 + pot e0, sum rot e0 + pot e1
//   A1..A3  = sum rot (e1^2 - e0^2, e0 e1, eps^2 / R^2),   B1..B3 the same with pot
//   L       = sum (s_y - s_x) A (40 (1 - p) + 10 p^2 - 2 p^3 / 3) e^-p,
//             p = |d|^2 / pse_eps^2
//   P, Q    = sum rot log R, sum pot log R
// give every output: 2 pi u = U, 2 pi v = V,
//   2 pi du/dx = 2 A2 + B1 + B3,   2 pi du/dy = A1 - A3 - 2 B2,
//   2 pi dv/dx = A1 + A3 - 2 B2,   2 pi dv/dy = -2 A2 - B1 + B3,
//   lap = L / (pi pse_eps^2), psi, phi = -P / 4 pi, -Q / 4 pi
// (R/2 taken from e1^2 and e0^2 pair by pair, so no large sums cancel).
// The FP64 pipe bounds the kernel, 64 clocks of a sub-partition per operation of a
// warp: 19 operations per pair (the differences, the sums and the two additions of
// the logarithm), everything between formed in integers beside them (swe_pair), against
// about 260 for the reference's operation order with its eight divisions, square root
// and library log and exp.  Quad level 5, vertices and faces: 19.6 ms in that order,
// 4.73 ms as moments in FP64 (55 operations), 1.64 ms now (0.88 of the pipe's rate).
constexpr int kSweNC = 11;

struct __align__(16) SweSrc {
  double x, y, rot, pot, s, area;
  int slot;
  int wild;  // (s_y - s_x) A may not be finite
  int pad[2];
};
// Not finite, or so large that a product of two such may not be.
__device__ __forceinline__ bool swe_wild(double v) {
  return (__double2hiint(v) & 0x7fffffff) >= (1023 + 500) << 20;
}

__global__ void k_swe_pack(View fx, const double* __restrict__ zeta, const double* __restrict__ sigma,
                           const double* __restrict__ area, const double* __restrict__ sfc,
                           const int* __restrict__ src2slot, int64_t ns, SweSrc* __restrict__ src) {
  const int64_t k = blockIdx.x * int64_t(blockDim.x) + threadIdx.x;
  if (k >= ns) return;
  const int64_t j = src2slot[k];
  SweSrc r;
  r.x = fx(j, 0);
  r.y = fx(j, 1);
  r.rot = dm(zeta[j], area[j]);
  r.pot = dm(sigma[j], area[j]);
  r.s = sfc[j];
  r.area = area[j];
  r.slot = int(j);
  r.wild = swe_wild(r.s) || swe_wild(r.area);
  r.pad[0] = r.pad[1] = 0;
  src[k] = r;
}
// A pair's factors: e = d / R, e1^2 - e0^2, e0 e1, eps^2 / R^2 (1 / R^2 itself overflows
// where the sums do not), log R and the smoothing kernel.
struct SwePair {
  double e0, e1, md, xy, ew, lg, pse;
};

// In FP64, for any values.
__device__ __noinline__ SwePair swe_pair_any(double d0, double d1, double epssq, double ipse2) {
  SwePair v;
  const double rsq = fma(d1, d1, d0 * d0), R = rsq + epssq, w = 1.0 / R, p = rsq * ipse2;
  v.e0 = d0 * w;
  v.e1 = d1 * w;
  v.md = fma(v.e1, v.e1, -(v.e0 * v.e0));
  v.xy = v.e0 * v.e1;
  v.ew = epssq * w * w;
  v.lg = log(R);
  v.pse = p >= 746.0 && p < INFINITY ? 0.0 : fma(p, fma(p, fma(p, -2.0 / 3, 10.0), -40.0), 40.0) * exp(-p);
  return v;
}

// eps^2 and 1 / pse_eps^2 for swe_pair: mantissas with bit 63 set (0 for eps = 0), and
// biased exponents; eps < 2^(ee - 1022).
struct SweScales {
  uint64_t e2, ip;
  int e2x, ipx, ee;
};
__device__ __forceinline__ SweScales swe_scales(double epssq, double ipse2) {
  SweScales c;
  c.e2x = int(unsigned(__double2hiint(epssq)) >> 20);
  c.ipx = int(unsigned(__double2hiint(ipse2)) >> 20);
  c.e2 = c.e2x > 0 ? f64_mantissa(epssq) << 11 : 0;
  c.ip = f64_mantissa(ipse2) << 11;
  c.ee = (c.e2x + 1023) / 2;
  // out of range: no pair is plain
  if (c.e2x > 1800 || c.ipx < 223 || c.ipx > 1823) c.ee = 4096;
  return c;
}

// In 64-bit fixed point: d over 2^(eE - 1085) for the larger exponent eE of d0, d1 and
// eps, so that |d|^2, R = |d|^2 + eps^2 and e1^2 - e0^2 keep 58 bits and more; e0, e1
// and their product from each component's own exponent, so that the smaller one loses
// nothing.  False for values it does not take: sizes outside 2^-240 .. 2^240, d below
// 2^-9 eps (whose last bits it would drop) but not 0, a component below 2^-200 of that
// but not 0, R beside 1.
__device__ __forceinline__ bool swe_pair(const F64Tables* __restrict__ tab, double d0, double d1,
                                         const SweScales& c, SwePair& v) {
  const unsigned h0 = unsigned(__double2hiint(d0)), h1 = unsigned(__double2hiint(d1));
  const int x0 = int(h0 >> 20 & 0x7ff), x1 = int(h1 >> 20 & 0x7ff), eb = max(x0, x1);
  const int eE = max(eb, c.ee);
  const uint64_t F0 = x0 > 0 ? f64_mantissa(d0) << 10 : 0, F1 = x1 > 0 ? f64_mantissa(d1) << 10 : 0;
  const int s0 = min(eE - x0, 63), s1 = min(eE - x1, 63);
  const uint64_t D0 = F0 >> s0, D1 = F1 >> s1;
  const uint64_t S = __umul64hi(D0, D0) + __umul64hi(D1, D1);  // |d|^2
  const uint64_t Q = S + (c.e2 >> min(2 * eE - 1020 - c.e2x, 63));  // R = Q 2^(2 eE - 2106)
  const int zq = __clzll(int64_t(Q | 1));
  const int xr = 2 * eE - 1020 - zq;
  const double R = __longlong_as_double(int64_t(f64_pack(Q << zq, xr)));
  const bool z0 = ((h0 << 1) | unsigned(__double2loint(d0))) == 0;
  const bool z1 = ((h1 << 1) | unsigned(__double2loint(d1))) == 0;
  if (unsigned(eE - 783) > 480u || (eE - eb > 9 && !(z0 && z1)) || (eE - x0 > 200 && !z0) ||
      (eE - x1 > 200 && !z1) || Q == 0 || !f64_log_plain(R))
    return false;
  const uint64_t W = f64_rcp_mantissa(R);
  const int er = int(unsigned(__double2hiint(R)) >> 20);
  const uint64_t E0 = __umul64hi(F0, W), E1 = __umul64hi(F1, W);  // |e| 2^(61 + er - x)
  const bool n0 = int(h0) < 0, n1 = int(h1) < 0;
  const int k0 = x0 - 61 - er, k1 = x1 - 61 - er;
  v.e0 = f64_value(E0, n0, k0);
  v.e1 = f64_value(E1, n1, k1);
  const uint64_t G0 = (2 * E0) >> s0, G1 = (2 * E1) >> s1;  // over the common exponent
  const int64_t md = int64_t(__umul64hi(G1, G1)) - int64_t(__umul64hi(G0, G0));
  v.md = f64_value(uint64_t(md < 0 ? -md : md), md < 0, 2 * (eE - 61 - er) + 62);
  v.xy = f64_value(__umul64hi(2 * E0, 2 * E1), n0 != n1, k0 + k1 + 62);
  const int kw = c.e2x - 1086 + 2 * (1023 - er);
  v.ew = f64_value(kw < -1000 ? 0 : __umul64hi(__umul64hi(W, W) << 2, c.e2), false, kw);
  v.lg = f64_log(tab, R);
  // p = |d|^2 / pse_eps^2
  const int zs = __clzll(int64_t(S | 1));
  const uint64_t pm = __umul64hi(S << zs, c.ip);
  const int zp = S == 0 ? 0 : __clzll(int64_t(pm));
  const int ep = S == 0 ? -1000 : 2 * eE - 2043 - zs + c.ipx - 1023 + 1 - zp;
  const uint64_t m = S == 0 ? uint64_t(1) << 63 : pm << zp;
  v.pse = 0.0;
  if (ep < 9 || (ep == 9 && m < 0xba80000000000000ull)) v.pse = f64_pse8(tab, m, ep);  // p < 746
  return true;
}

// COLL: collocated targets, the source in the target's own slot is skipped.
template <bool COLL>
__global__ void __launch_bounds__(kSweNT) k_swe_plane(View tx, const double* __restrict__ ts,
                                                      int64_t nt, const SweSrc* __restrict__ src,
                                                      int64_t ns, int64_t chunk_len, double epssq,
                                                      double ipse2, const F64Tables* __restrict__ tab,
                                                      double* __restrict__ part, int64_t tpad) {
  __shared__ SweSrc tile[kSweTile64];
  const int64_t i = blockIdx.x * int64_t(blockDim.x) + threadIdx.x;
  const int64_t c = blockIdx.y;
  const int64_t j0 = c * chunk_len, j1 = ns < j0 + chunk_len ? ns : j0 + chunk_len;
  const bool valid = i < nt;
  const double x0 = valid ? tx(i, 0) : 0.0, x1 = valid ? tx(i, 1) : 0.0;
  const double si = valid ? ts[i] : 0.0;
  const bool wild = swe_wild(si);
  const SweScales sc = swe_scales(epssq, ipse2);
  double r[kSweNC];
#pragma unroll
  for (int k = 0; k < kSweNC; ++k) r[k] = 0.0;
  for (int64_t t0 = j0; t0 < j1; t0 += kSweTile64) {
    const int m = int(j1 - t0 < kSweTile64 ? j1 - t0 : kSweTile64);
    __syncthreads();
    for (int q = threadIdx.x; q < m * int(sizeof(SweSrc) / 16); q += blockDim.x)
      reinterpret_cast<double2*>(tile)[q] = reinterpret_cast<const double2*>(src + t0)[q];
    __syncthreads();
    if (!valid) continue;
#pragma unroll 1
    for (int q = 0; q < m; ++q) {
      const SweSrc& y = tile[q];
      if (COLL && y.slot == i) continue;
      const double d0 = x0 - y.x, d1 = x1 - y.y;
      SwePair v;
      if (!swe_pair(tab, d0, d1, sc, v)) v = swe_pair_any(d0, d1, epssq, ipse2);
      r[0] = fma(-y.rot, v.e1, fma(y.pot, v.e0, r[0]));
      r[1] = fma(y.rot, v.e0, fma(y.pot, v.e1, r[1]));
      r[2] = fma(y.rot, v.md, r[2]);
      r[3] = fma(y.rot, v.xy, r[3]);
      r[4] = fma(y.rot, v.ew, r[4]);
      r[5] = fma(y.pot, v.md, r[5]);
      r[6] = fma(y.pot, v.xy, r[6]);
      r[7] = fma(y.pot, v.ew, r[7]);
      // (0 times a value that is not finite is NaN)
      if (v.pse != 0.0 || wild || y.wild) r[8] = fma((y.s - si) * y.area, v.pse, r[8]);
      r[9] = fma(y.rot, v.lg, r[9]);
      r[10] = fma(y.pot, v.lg, r[10]);
    }
  }
  if (!valid) return;
#pragma unroll
  for (int k = 0; k < kSweNC; ++k) part[(c * kSweNC + k) * tpad + i] = r[k];
}

struct SweOut {
  View u;
  double *ddot, *du1dx1, *du1dx2, *du2dx1, *du2dx2, *laps, *psi, *phi;
  int do_velocity;
};

// Outputs of one target from its velocity sums (times 2 pi), gradients,
// Laplacian and stream/potential functions.
__device__ __forceinline__ void swe_write(const SweOut& o, int64_t i, double u, double v, double g00,
                                          double g01, double g10, double g11, double lap, double psi,
                                          double phi) {
  if (o.do_velocity) {
    o.u(i, 0) = u;
    o.u(i, 1) = v;
  }
  // square(du/dx) + 2 du/dy dv/dx + square(dv/dy)
  o.ddot[i] = da(da(dm(g00, g00), dm(dm(2.0, g01), g10)), dm(g11, g11));
  o.du1dx1[i] = g00;
  o.du1dx2[i] = g01;
  o.du2dx1[i] = g10;
  o.du2dx2[i] = g11;
  o.laps[i] = lap;
  o.psi[i] = psi;
  o.phi[i] = phi;
}

__global__ void k_swe_out(const double* __restrict__ part, int64_t tpad, int64_t nt, double pse_eps,
                          SweOut o) {
  const int64_t i = blockIdx.x * int64_t(blockDim.x) + threadIdx.x;
  if (i >= nt) return;
  double s[kSweNC];
#pragma unroll
  for (int k = 0; k < kSweNC; ++k) s[k] = part[k * tpad + i];
  const double i2pi = 0.5 / kPI, i4pi = 0.25 / kPI;
  const double ea = s[4], eb = s[7], a2 = 2.0 * s[3], b2 = 2.0 * s[6];
  swe_write(o, i, s[0] * i2pi, s[1] * i2pi, (a2 + s[5] + eb) * i2pi, (s[2] - ea - b2) * i2pi,
            (s[2] + ea - b2) * i2pi, (eb - a2 - s[5]) * i2pi, s[8] / (kPI * pse_eps * pse_eps),
            -s[9] * i4pi, -s[10] * i4pi);
}

// ---- planar SWE sums, FP32 compensated (context precision LPM_FP32C) ------
// With d = x - y, R = |d|^2 + eps^2, r = 1/R, a = rot r, b = pot r, every
// output is a sum of per-pair moments (15 per target):
//   w0..3 = sum a d0, a d1, b d0, b d1      w4, w5 = sum a, sum b
//   w6..8 = sum a r (d0^2, d0 d1, d1^2)     w9..11 = the same with b
//   w12 = sum (s_y - s_x) A lapPSE(|d|^2 / pse_eps^2)
//   w13, w14 = sum rot lg2 R, sum pot lg2 R
// and the FP64 epilogue forms u = (-w1 + w2) / 2pi, v = (w0 + w3) / 2pi,
// du/dx = (w7 - w9) / pi + w5 / 2pi, du/dy = (w8 - w10) / pi - w4 / 2pi,
// dv/dx = (-w6 - w10) / pi + w4 / 2pi, dv/dy = (-w7 - w11) / pi + w5 / 2pi,
// lap = w12 / (pi pse_eps^2), psi, phi = -(ln 2 / 4pi) w13, w14.  The PSE
// kernel uses |d|^2 directly (the reference's sqrt then square is the
// identity).  Positions and surface heights are split into FP32 hi + lo parts
// (d and s_y - s_x are small differences of O(1) values).  Three MUFU
// results (reciprocal, log2, exp2) and ~45 FP32 operations per pair, two
// sources per packed f32x2 instruction (pair k holds sources 2k, 2k + 1; an
// odd count ends with a zero-strength, zero-area source), the sums kept per
// lane over a 256-source tile and then merged by TwoSum.
constexpr int kPl32NC = 15;

struct __align__(16) PlPair32 {
  float4 hxy;  // x hi of sources 2k, 2k + 1; y hi
  float4 lxy;  // x lo; y lo
  float4 rp;   // rot; pot
  float4 as;   // area; surface hi
  float4 sl;   // surface lo; slot (int bits)
};

__global__ void k_swe_plane32_pack(View fx, const double* __restrict__ zeta,
                                   const double* __restrict__ sigma,
                                   const double* __restrict__ area, const double* __restrict__ sfc,
                                   const int* __restrict__ src2slot, int64_t ns,
                                   PlPair32* __restrict__ src) {
  const int64_t k = blockIdx.x * int64_t(blockDim.x) + threadIdx.x;
  if (k >= (ns + 1) / 2) return;
  float v[2][9] = {};
  int sl[2] = {-1, -1};
#pragma unroll
  for (int e = 0; e < 2; ++e) {
    if (2 * k + e >= ns) break;
    const int64_t j = src2slot[2 * k + e];
    const double x = fx(j, 0), y = fx(j, 1), sv = sfc[j];
    const float xh = float(x), yh = float(y), sh = float(sv);
    v[e][0] = xh;
    v[e][1] = yh;
    v[e][2] = float(x - xh);
    v[e][3] = float(y - yh);
    v[e][4] = float(zeta[j] * area[j]);
    v[e][5] = float(sigma[j] * area[j]);
    v[e][6] = float(area[j]);
    v[e][7] = sh;
    v[e][8] = float(sv - sh);
    sl[e] = int(j);
  }
  PlPair32 r;
  r.hxy = make_float4(v[0][0], v[1][0], v[0][1], v[1][1]);
  r.lxy = make_float4(v[0][2], v[1][2], v[0][3], v[1][3]);
  r.rp = make_float4(v[0][4], v[1][4], v[0][5], v[1][5]);
  r.as = make_float4(v[0][6], v[1][6], v[0][7], v[1][7]);
  r.sl = make_float4(v[0][8], v[1][8], __int_as_float(sl[0]), __int_as_float(sl[1]));
  src[k] = r;
}

// One pair record against one target.  COLL: face targets; the source in the
// target's own slot is skipped (its reciprocal and logarithm are replaced by
// 0, and its PSE term is 0: d = 0 and s_y - s_x = 0).  TAIL: the record may
// hold the zero-strength dummy (slot -1, at the origin, which can coincide
// with a target), whose reciprocal and logarithm are zeroed the same way.
struct Pl32Target {
  u64 x0h, x1h, sh, x0l, x1l, sl, e2, ipse2;
  int64_t i;
};

template <bool COLL, bool TAIL>
__device__ __forceinline__ void pl32_pair(const PlPair32& s, const Pl32Target& t,
                                          u64 (&w)[kPl32NC]) {
  const u64 d0 = add2(sub2(t.x0h, pk2(s.hxy.x, s.hxy.y)), sub2(t.x0l, pk2(s.lxy.x, s.lxy.y)));
  const u64 d1 = add2(sub2(t.x1h, pk2(s.hxy.z, s.hxy.w)), sub2(t.x1l, pk2(s.lxy.z, s.lxy.w)));
  const u64 dd = fma2(d0, d0, mul2(d1, d1));
  float qa, qb;
  upk2(add2(dd, t.e2), qa, qb);
  float ra = rcp_approx(qa), rb = rcp_approx(qb);
  float la = lg2_approx(qa), lb = lg2_approx(qb);
  if (COLL || TAIL) {
    const int sa = __float_as_int(s.sl.z), sb = __float_as_int(s.sl.w);
    const bool ska = (COLL && sa == t.i) || (TAIL && sa < 0);
    const bool skb = (COLL && sb == t.i) || (TAIL && sb < 0);
    ra = ska ? 0.f : ra;
    la = ska ? 0.f : la;
    rb = skb ? 0.f : rb;
    lb = skb ? 0.f : lb;
  }
  const u64 r = pk2(ra, rb), L = pk2(la, lb);
  const u64 p2 = mul2(dd, t.ipse2);
  float ea, eb;
  upk2(mul2(p2, pk2(-1.4426950408889634f, -1.4426950408889634f)), ea, eb);
  float xa, xb;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(xa) : "f"(ea));
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(xb) : "f"(eb));
  const u64 poly = fma2(fma2(fma2(pk2(-2.f / 3.f, -2.f / 3.f), p2, pk2(10.f, 10.f)), p2,
                             pk2(-40.f, -40.f)),
                        p2, pk2(40.f, 40.f));
  const u64 ds = add2(sub2(pk2(s.as.z, s.as.w), t.sh), sub2(pk2(s.sl.x, s.sl.y), t.sl));
  const u64 rot = pk2(s.rp.x, s.rp.y), pot = pk2(s.rp.z, s.rp.w);
  const u64 a = mul2(rot, r), b = mul2(pot, r);
  const u64 a2 = mul2(a, r), b2 = mul2(b, r);
  w[0] = fma2(a, d0, w[0]);
  w[1] = fma2(a, d1, w[1]);
  w[2] = fma2(b, d0, w[2]);
  w[3] = fma2(b, d1, w[3]);
  w[4] = add2(w[4], a);
  w[5] = add2(w[5], b);
  const u64 ad0 = mul2(a2, d0), ad1 = mul2(a2, d1), bd0 = mul2(b2, d0), bd1 = mul2(b2, d1);
  w[6] = fma2(ad0, d0, w[6]);
  w[7] = fma2(ad0, d1, w[7]);
  w[8] = fma2(ad1, d1, w[8]);
  w[9] = fma2(bd0, d0, w[9]);
  w[10] = fma2(bd0, d1, w[10]);
  w[11] = fma2(bd1, d1, w[11]);
  w[12] = fma2(mul2(ds, pk2(s.as.x, s.as.y)), mul2(poly, pk2(xa, xb)), w[12]);
  w[13] = fma2(rot, L, w[13]);
  w[14] = fma2(pot, L, w[14]);
}

template <bool COLL>
__global__ void __launch_bounds__(kSweNT) k_swe_plane32(View tx, const double* __restrict__ ts,
                                                        int64_t nt, const PlPair32* __restrict__ src,
                                                        int64_t ns, int64_t chunk_len, float e2,
                                                        float ipse2, double* __restrict__ part,
                                                        int64_t tpad) {
  __shared__ PlPair32 tile[kSweTile / 2];
  const int64_t i = blockIdx.x * int64_t(kSweNT) + threadIdx.x;
  const int64_t c = blockIdx.y;
  const int64_t j0 = c * chunk_len, j1 = ns < j0 + chunk_len ? ns : j0 + chunk_len;
  const bool valid = i < nt;
  const double X0 = valid ? tx(i, 0) : 0.0, X1 = valid ? tx(i, 1) : 0.0;
  const double SX = valid ? ts[i] : 0.0;
  const float x0h = float(X0), x1h = float(X1), sxh = float(SX);
  const float x0l = float(X0 - x0h), x1l = float(X1 - x1h), sxl = float(SX - sxh);
  const Pl32Target t{pk2(x0h, x0h), pk2(x1h, x1h), pk2(sxh, sxh), pk2(x0l, x0l),
                     pk2(x1l, x1l), pk2(sxl, sxl), pk2(e2, e2),  pk2(ipse2, ipse2), i};
  float S[kPl32NC], C[kPl32NC];
#pragma unroll
  for (int k = 0; k < kPl32NC; ++k) S[k] = C[k] = 0.f;
  for (int64_t t0 = j0; t0 < j1; t0 += kSweTile) {  // t0 is even: chunks are whole tiles
    const int m = int(j1 - t0 < kSweTile ? j1 - t0 : kSweTile);
    const int mp = (m + 1) / 2;
    __syncthreads();
    for (int q = threadIdx.x; q < mp; q += kSweNT) tile[q] = src[t0 / 2 + q];
    __syncthreads();
    if (!valid) continue;
    u64 w[kPl32NC];
#pragma unroll
    for (int k = 0; k < kPl32NC; ++k) w[k] = 0ull;
#pragma unroll 2
    for (int q = 0; q < m / 2; ++q) pl32_pair<COLL, false>(tile[q], t, w);
    if (m & 1) pl32_pair<COLL, true>(tile[mp - 1], t, w);  // the dummy's pair
#pragma unroll
    for (int k = 0; k < kPl32NC; ++k) {
      float a, b;
      upk2(w[k], a, b);
      two_sum_acc(S[k], C[k], a);
      two_sum_acc(S[k], C[k], b);
    }
  }
  if (!valid) return;
#pragma unroll
  for (int k = 0; k < kPl32NC; ++k) part[(c * kPl32NC + k) * tpad + i] = double(S[k]) + double(C[k]);
}

__global__ void k_swe_plane32_out(const double* __restrict__ part, int64_t tpad, int64_t nt, double pse_eps, SweOut o) {
  const int64_t i = blockIdx.x * int64_t(blockDim.x) + threadIdx.x;
  if (i >= nt) return;
  double w[kPl32NC];
#pragma unroll
  for (int k = 0; k < kPl32NC; ++k) w[k] = part[k * tpad + i];
  const double ipi = 1.0 / kPI, i2pi = 0.5 / kPI;
  const double k = -0.6931471805599453 / (4 * kPI);
  swe_write(o, i, (w[2] - w[1]) * i2pi, (w[0] + w[3]) * i2pi, (w[7] - w[9]) * ipi + w[5] * i2pi,
            (w[8] - w[10]) * ipi - w[4] * i2pi, -(w[6] + w[10]) * ipi + w[4] * i2pi,
            -(w[7] + w[11]) * ipi + w[5] * i2pi, w[12] * ipi / (pse_eps * pse_eps), k * w[13],
            k * w[14]);
}

// ---- spherical SWE sums ----------------------------------------------------
// Pair term (sphere_swe_velocity_sums, :335-373) with s = x.y,
// D = (1 - s) + eps^2, c = x cross y, rot = -zeta A, pot = -sigma A, and
// P = I - x x^T:
//   u += c rot / (4 pi D) + P y pot / (4 pi D)
//   M += gkz rot + gks pot, where the reference's polynomials for grad_kzeta
//   and grad_ksigma (:114-325) equal, over 4 pi D^2 (gkz identically, gks on
//   the unit sphere),
//     gkz = D [y]x + c v^T,          v = (1 + eps^2) x - y
//     gks = -v w^T - D s P,          w = P y = y - s x
//   (w - D x = -v because s + D = 1 + eps^2).
// Sums over sources are taken in the target's frame (t1, t2, n), x = rho n: with
// p_a = t_a.(x - y), sz, ss = rot, pot / (4 pi D) and R, Q = rot, pot / (4 pi D^2),
// c = rho (p2, -p1, 0), w = (-p1, -p2, k yn) and v = (p1, p2, rho D - k yn) for
// k = 1 - |x|^2 and yn = s / rho, so the 17 sums
//   sz p, ss p;  R, Q (p1 p1, p1 p2, p2 p2);  sz s, ss s;
//   R s p, Q s p, Q s^2 (times k: targets off the unit sphere)
// give u and M (sph_assemble).  A sum along x would be n / sqrt(n) times larger
// than the tangential ones it is added to in fixed axes, whose roundings then
// stay when x is projected out (same-sign strengths: errors 30 times larger), and
// eps^2 enters no difference of sums.  t_a.x is not 0 but about 1e-16: p_a leaves it
// out exactly (tau_a), as it would add up over the sources.
// FP64: s and D = (1 - s) + eps^2 unfused in the reference's order (D is
// the ill-conditioned quantity: a one-ulp change of s moves a near pair's D by
// ~1e-16 / D relative), everything after it contracted, one reciprocal of D per
// pair in integers (f64math.cuh).  The FP64 pipe bounds the kernel: 44 operations
// per pair (66 in the form that added c v^T, v w^T, u term by term in fixed axes, 48
// as moments of x - y in fixed axes): icosahedral level 5, vertices and faces, 96.5 /
// 68.5 / 61.4 ms, level 2, where chunks of 8 to 64 sources fill the SMs, 0.143 ms.
constexpr int kSphNC = 17;

struct __align__(16) SphSrc {
  double x, y, z, rot, pot;  // strengths over 4 pi
  int slot, pad;
};

// a.b exactly to about 1e-31, rounded to FP64.
__device__ __forceinline__ double exact_dot(const double (&a)[3], const double (&b)[3], double s) {
  double e = 0.0;
#pragma unroll
  for (int c = 0; c < 3; ++c) {
    const double p = dm(a[c], b[c]), pe = fma(a[c], b[c], -p);
    const double t = da(s, p), bb = ds(t, s);
    e += ds(s, ds(t, bb)) + ds(p, bb) + pe;
    s = t;
  }
  return s + e;
}

// A target's frame, once per call (about 200 FP64 operations, as many as five pairs,
// and a chunk may hold eight): t1, t2, tau1, tau2, tau1 / rho^2, tau2 / rho^2 for the
// pair kernel; n, rho, 1 - rho^2 for the assembly.  At x = 0 any frame, rho = 0.
enum : int { kT1 = 0, kT2 = 3, kTau = 6, kTauR = 8, kN = 10, kRho = 13, kDef = 14, kSphFrame = 15 };

__device__ __forceinline__ void sph_frame(const double (&x)[3], double (&f)[kSphFrame]) {
  const double mx[3] = {-x[0], -x[1], -x[2]};
  f[kDef] = exact_dot(mx, x, 1.0);
  double rho = sqrt(exact_dot(x, x, 0.0));
  const bool zero = rho < 0x1p-300;
  if (zero) rho = 0.0;
  f[kRho] = rho;
  const double ir = 1.0 / rho;
  double n[3];
#pragma unroll
  for (int a = 0; a < 3; ++a) f[kN + a] = n[a] = zero ? (a == 2 ? 1.0 : 0.0) : x[a] * ir;
  const double sg = n[2] >= 0.0 ? 1.0 : -1.0, q = -1.0 / (sg + n[2]), b = n[0] * n[1] * q;
  const double t1[3] = {1.0 + sg * n[0] * n[0] * q, sg * b, -sg * n[0]};
  const double t2[3] = {b, sg + n[1] * n[1] * q, -n[1]};
  const double tau[2] = {exact_dot(t1, x, 0.0), exact_dot(t2, x, 0.0)};
#pragma unroll
  for (int a = 0; a < 3; ++a) f[kT1 + a] = t1[a], f[kT2 + a] = t2[a];
#pragma unroll
  for (int a = 0; a < 2; ++a) {
    f[kTau + a] = zero ? 0.0 : tau[a];
    f[kTauR + a] = zero ? 0.0 : tau[a] * (ir * ir);
  }
}

// Source records, and in the blocks after them the targets' frames.
__global__ void k_swe_sphere_pack(View fx, const double* __restrict__ zeta,
                                  const double* __restrict__ sigma, const double* __restrict__ area,
                                  const int* __restrict__ src2slot, int64_t ns,
                                  SphSrc* __restrict__ src, View tx, int64_t nt, int64_t tpad,
                                  double* __restrict__ fr) {
  const int64_t src_blocks = (ns + blockDim.x - 1) / blockDim.x;
  if (int64_t(blockIdx.x) >= src_blocks) {
    const int64_t i = (blockIdx.x - src_blocks) * int64_t(blockDim.x) + threadIdx.x;
    if (i >= nt) return;
    const double x[3] = {tx(i, 0), tx(i, 1), tx(i, 2)};
    double f[kSphFrame];
    sph_frame(x, f);
#pragma unroll
    for (int k = 0; k < kSphFrame; ++k) fr[k * tpad + i] = f[k];
    return;
  }
  const int64_t k = blockIdx.x * int64_t(blockDim.x) + threadIdx.x;
  if (k >= ns) return;
  const int64_t j = src2slot[k];
  SphSrc r;
  r.x = fx(j, 0);
  r.y = fx(j, 1);
  r.z = fx(j, 2);
  const double inv4pi = 1.0 / (4 * kPI);
  r.rot = -zeta[j] * area[j] * inv4pi;
  r.pot = -sigma[j] * area[j] * inv4pi;
  r.slot = int(j);
  r.pad = 0;
  src[k] = r;
}

// COLL: collocated targets, the source in the target's own slot is skipped.
template <bool COLL>
__global__ void __launch_bounds__(kSweNT) k_swe_sphere(View tx, int64_t nt,
                                                       const double* __restrict__ fr,
                                                       const SphSrc* __restrict__ src, int64_t ns,
                                                       int64_t chunk_len, double epssq,
                                                       double* __restrict__ part, int64_t tpad) {
  __shared__ SphSrc tile[kSweTile64];
  const int64_t i = blockIdx.x * int64_t(blockDim.x) + threadIdx.x;
  const int64_t c = blockIdx.y;
  const int64_t j0 = c * chunk_len, j1 = ns < j0 + chunk_len ? ns : j0 + chunk_len;
  const bool valid = i < nt;
  double x[3];
#pragma unroll
  for (int a = 0; a < 3; ++a) x[a] = valid ? tx(i, a) : 0.0;
  double f[kN];
#pragma unroll
  for (int k = 0; k < kN; ++k) f[k] = valid ? fr[k * tpad + i] : 0.0;
  const bool zero = valid && fr[kRho * tpad + i] == 0.0;
  double r[kSphNC];
#pragma unroll
  for (int k = 0; k < kSphNC; ++k) r[k] = 0.0;
  for (int64_t t0 = j0; t0 < j1; t0 += kSweTile64) {
    const int m = int(j1 - t0 < kSweTile64 ? j1 - t0 : kSweTile64);
    __syncthreads();
    for (int q = threadIdx.x; q < m * int(sizeof(SphSrc) / 16); q += blockDim.x)
      reinterpret_cast<double2*>(tile)[q] = reinterpret_cast<const double2*>(src + t0)[q];
    __syncthreads();
    if (!valid) continue;
#pragma unroll 1
    for (int q = 0; q < m; ++q) {
      const SphSrc& y = tile[q];
      if (COLL && y.slot == i) continue;
      // x.y unfused in the reference's order: 1 - s cancels, and its rounding
      // is the reference's
      const double s = da(da(dm(x[0], y.x), dm(x[1], y.y)), dm(x[2], y.z));
      const double D = da(ds(1.0, s), epssq);
      const double rd = f64_inv(D);
      const double d[3] = {x[0] - y.x, x[1] - y.y, x[2] - y.z};
      // t_a.d less its part along x, tau_a (1 - s / rho^2)
      const double p1 = fma(f[kTauR], s, fma(f[0], d[0], fma(f[1], d[1], fma(f[2], d[2], -f[kTau]))));
      const double p2 = fma(f[kTauR + 1], s, fma(f[3], d[0], fma(f[4], d[1], fma(f[5], d[2], -f[kTau + 1]))));
      const double sz = y.rot * rd, ss = y.pot * rd;
      const double R = sz * rd, Q = ss * rd;
      const double r1 = R * p1, r2 = R * p2, q1 = Q * p1, q2 = Q * p2;
      double sn = s;  // rho yn; yn at x = 0
      if (zero) sn = y.z;
      r[0] = fma(sz, p1, r[0]);
      r[1] = fma(sz, p2, r[1]);
      r[2] = fma(ss, p1, r[2]);
      r[3] = fma(ss, p2, r[3]);
      r[4] = fma(r1, p1, r[4]);
      r[5] = fma(r1, p2, r[5]);
      r[6] = fma(r2, p2, r[6]);
      r[7] = fma(q1, p1, r[7]);
      r[8] = fma(q1, p2, r[8]);
      r[9] = fma(q2, p2, r[9]);
      r[10] = fma(sz, sn, r[10]);
      r[11] = fma(ss, sn, r[11]);
      r[12] = fma(r1, sn, r[12]);
      r[13] = fma(r2, sn, r[13]);
      r[14] = fma(q1, sn, r[14]);
      r[15] = fma(q2, sn, r[15]);
      r[16] = fma(Q * sn, sn, r[16]);
    }
  }
  if (!valid) return;
#pragma unroll
  for (int k = 0; k < kSphNC; ++k) part[(c * kSphNC + k) * tpad + i] = r[k];
}

// u and M of one target in its frame, then in the caller's axes.
__device__ __forceinline__ void sph_assemble(const double (&f)[kSphFrame], const double (&s)[kSphNC],
                                             double (&u)[3], double (&M)[9]) {
  const double rho = f[kRho], k = f[kDef];
  const bool zero = rho == 0.0;
  const double ir = zero ? 1.0 : 1.0 / rho;  // yn = ir sn
  const double kir = k * ir, rk = zero ? 0.0 : k;
  const double Yn = s[10] * ir, G = zero ? 0.0 : s[11];  // sum sz yn, sum ss x.y
  const double ul[3] = {rho * s[1] - s[2], -rho * s[0] - s[3], kir * s[11]};
  // sum sz y = (-s0, -s1, Yn); P = diag(1, 1, k)
  // (R c_a v_n = +-rho R (rho D - k yn) p; Q v_n = rho ss - k Q yn)
  const double vn1 = rho * s[2] - kir * s[14], vn2 = rho * s[3] - kir * s[15];
  const double L[9] = {
      rho * s[5] + s[7] - G,  rho * s[6] + s[8] - Yn,  rho * rho * s[1] - rk * s[13] - kir * s[14] - s[1],
      -rho * s[4] + s[8] + Yn, -rho * s[5] + s[9] - G, -rho * rho * s[0] + rk * s[12] - kir * s[15] + s[0],
      vn1 + s[1],             vn2 - s[0],              -kir * (rho * s[11] - kir * s[16]) - G * k};
#pragma unroll
  for (int a = 0; a < 3; ++a) u[a] = ul[0] * f[kT1 + a] + ul[1] * f[kT2 + a] + ul[2] * f[kN + a];
#pragma unroll
  for (int a = 0; a < 3; ++a) {
    double h[3];  // row a of (F L)
#pragma unroll
    for (int q = 0; q < 3; ++q) h[q] = f[kT1 + a] * L[q] + f[kT2 + a] * L[3 + q] + f[kN + a] * L[6 + q];
#pragma unroll
    for (int b = 0; b < 3; ++b) M[3 * a + b] = h[0] * f[kT1 + b] + h[1] * f[kT2 + b] + h[2] * f[kN + b];
  }
}

__global__ void k_swe_sphere_out(const double* __restrict__ part, int64_t tpad,
                                 const double* __restrict__ fr, int64_t nt, View u,
                                 double* __restrict__ ddot, double* __restrict__ grad,
                                 int do_velocity) {
  const int64_t i = blockIdx.x * int64_t(blockDim.x) + threadIdx.x;
  if (i >= nt) return;
  double s[kSphNC], f[kSphFrame], v[3], M[9];
#pragma unroll
  for (int k = 0; k < kSphNC; ++k) s[k] = part[k * tpad + i];
#pragma unroll
  for (int k = 0; k < kSphFrame; ++k) f[k] = fr[k * tpad + i];
  sph_assemble(f, s, v, M);
  if (do_velocity)
#pragma unroll
    for (int a = 0; a < 3; ++a) u(i, a) = v[a];
  // sum_ij M_ij M_ji in the functors' loop order
  double dsum = 0.0;
#pragma unroll
  for (int a = 0; a < 3; ++a)
#pragma unroll
    for (int b = 0; b < 3; ++b) dsum = da(dsum, dm(M[3 * a + b], M[3 * b + a]));
  ddot[i] = dsum;
  if (grad)
#pragma unroll
    for (int k = 0; k < 9; ++k) grad[9 * i + k] = M[k];
}

// ---- spherical SWE sums, FP32 compensated (context precision LPM_FP32C) ----
// Chord form: with d = x - y for unit vectors, 1 - x.y = |d|^2 / 2, so
// D = q / 2 with q = |d|^2 + 2 eps^2, and c = x cross y = d cross x,
// v = eps^2 x + d, w = P y = -P d.  Writing rs, ps = rot, pot / (2 pi) and
// r = 1/q, the pair scalars are sz = rs r, ss = ps r (= rot, pot / (4 pi D))
// and R = 2 sz r, Q = 2 ss r (= rot, pot / (4 pi D^2)).  Every term is then a
// moment of d, summed per target (27 sums):
//   A = sum sz d, B = sum ss d, U1 = sum R d, V1 = sum Q d,
//   U2 = sum R d d^T, V2 = sum Q d d^T (symmetric), Z = sum sz, G = sum ss,
//   H = sum ss |d|^2,
// and the epilogue (FP64) assembles
//   u = A x x - P B
//   M = eps^2 (U1 x x) x^T + [U2 columns] x x + eps^2 x (P V1)^T + V2 P
//       + [Z x - A]x - (G - H/2) P.
// Positions are split into FP32 hi + lo parts so that d = (xh - yh) +
// (xl - yl) carries its own FP32 rounding, not the positions' (near pairs
// dominate the gradient: their |d| shrinks with the mesh).  Per pair: 50 FP32
// operations and one MUFU reciprocal (the strengths are stored doubled, as
// rot, pot / pi, so that R, Q = sz r, ss r need no doubling; the epilogue
// halves the sums of sz and ss, exactly).  Two sources per packed f32x2
// instruction: pair k of the packed array holds sources 2k and 2k + 1 (an odd
// count ends with a zero-strength source at the origin, whose terms are
// exactly 0), each thread owns one target, and the 27 sums are kept per lane
// (even and odd sources) over a 256-source tile; the two lanes' tile
// partials are then added into FP64 running sums in shared memory (which
// frees the registers the packed sums need).
constexpr int kSph32NC = 27;  // A3 B3 U1[3] V1[3] U2[6] V2[6] Z G H

struct __align__(16) SphPair32 {
  float4 hxy;  // x hi of sources 2k, 2k + 1; y hi of 2k, 2k + 1
  float4 hzr;  // z hi; rot / pi (twice rs: see above)
  float4 lxy;  // x lo (x - x hi); y lo
  float4 lzp;  // z lo; pot / pi
};

__global__ void k_swe_sphere32_pack(View fx, const double* __restrict__ zeta,
                                    const double* __restrict__ sigma,
                                    const double* __restrict__ area,
                                    const int* __restrict__ src2slot, int64_t ns,
                                    SphPair32* __restrict__ src, int2* __restrict__ slot) {
  const int64_t k = blockIdx.x * int64_t(blockDim.x) + threadIdx.x;
  if (k >= (ns + 1) / 2) return;
  const double inv_pi = 1.0 / kPI;  // strengths stored doubled: rot, pot / pi
  float h[2][4] = {}, l[2][4] = {};
  int sl[2] = {-1, -1};
#pragma unroll
  for (int e = 0; e < 2; ++e) {
    if (2 * k + e >= ns) break;
    const int64_t j = src2slot[2 * k + e];
    const double x = fx(j, 0), y = fx(j, 1), z = fx(j, 2);
    h[e][0] = float(x);
    h[e][1] = float(y);
    h[e][2] = float(z);
    h[e][3] = float(-zeta[j] * area[j] * inv_pi);
    l[e][0] = float(x - double(h[e][0]));
    l[e][1] = float(y - double(h[e][1]));
    l[e][2] = float(z - double(h[e][2]));
    l[e][3] = float(-sigma[j] * area[j] * inv_pi);
    sl[e] = int(j);
  }
  SphPair32 r;
  r.hxy = make_float4(h[0][0], h[1][0], h[0][1], h[1][1]);
  r.hzr = make_float4(h[0][2], h[1][2], h[0][3], h[1][3]);
  r.lxy = make_float4(l[0][0], l[1][0], l[0][1], l[1][1]);
  r.lzp = make_float4(l[0][2], l[1][2], l[0][3], l[1][3]);
  src[k] = r;
  slot[k] = make_int2(sl[0], sl[1]);
}

// COLL: face targets; the source in the target's own slot is skipped (its
// reciprocal is replaced by 0, which zeroes every term of the pair).
template <bool COLL>
__global__ void __launch_bounds__(kSweNT, 4) k_swe_sphere32(View tx, int64_t nt,
                                                            const SphPair32* __restrict__ src,
                                                            const int2* __restrict__ slot,
                                                            int64_t ns, int64_t chunk_len, float c0,
                                                            double* __restrict__ part,
                                                            int64_t tpad) {
  __shared__ SphPair32 tile[kSweTile / 2];
  __shared__ int2 tslot[COLL ? kSweTile / 2 : 1];
  __shared__ double acc[kSph32NC][kSweNT];
  const int tid = threadIdx.x;
  const int64_t i = blockIdx.x * int64_t(kSweNT) + tid;
  const int64_t c = blockIdx.y;
  const int64_t j0 = c * chunk_len, j1 = ns < j0 + chunk_len ? ns : j0 + chunk_len;
  const bool valid = i < nt;
  u64 XH[3], XL[3];
#pragma unroll
  for (int a = 0; a < 3; ++a) {
    const double v = valid ? tx(i, a) : 0.0;
    const float h = float(v), l = float(v - double(h));
    XH[a] = pk2(h, h);
    XL[a] = pk2(l, l);
  }
  const u64 C02 = pk2(c0, c0);
#pragma unroll
  for (int k = 0; k < kSph32NC; ++k) acc[k][tid] = 0.0;
  for (int64_t t0 = j0; t0 < j1; t0 += kSweTile) {  // t0 is even: chunks are whole tiles
    const int m = int(j1 - t0 < kSweTile ? j1 - t0 : kSweTile);
    const int mp = (m + 1) / 2;
    __syncthreads();
    for (int q = tid; q < mp; q += kSweNT) {
      tile[q] = src[t0 / 2 + q];
      if (COLL) tslot[q] = slot[t0 / 2 + q];
    }
    __syncthreads();
    if (!valid) continue;
    u64 w[kSph32NC];
#pragma unroll
    for (int k = 0; k < kSph32NC; ++k) w[k] = 0ull;
#pragma unroll 2
    for (int q = 0; q < mp; ++q) {
      const SphPair32 s = tile[q];
      const u64 d0 = add2(sub2(XH[0], pk2(s.hxy.x, s.hxy.y)), sub2(XL[0], pk2(s.lxy.x, s.lxy.y)));
      const u64 d1 = add2(sub2(XH[1], pk2(s.hxy.z, s.hxy.w)), sub2(XL[1], pk2(s.lxy.z, s.lxy.w)));
      const u64 d2 = add2(sub2(XH[2], pk2(s.hzr.x, s.hzr.y)), sub2(XL[2], pk2(s.lzp.x, s.lzp.y)));
      const u64 dd = fma2(d0, d0, fma2(d1, d1, mul2(d2, d2)));
      float qa, qb;
      upk2(add2(dd, C02), qa, qb);
      float ra = rcp_approx(qa), rb = rcp_approx(qb);
      if (COLL) {
        const int2 sl = tslot[q];
        ra = sl.x == i ? 0.f : ra;
        rb = sl.y == i ? 0.f : rb;
      }
      const u64 r = pk2(ra, rb);
      // sz, ss are twice the pair scalars (the strengths are stored doubled),
      // so R, Q = sz r, ss r; the sums of sz and ss are halved in the epilogue
      const u64 sz = mul2(pk2(s.hzr.z, s.hzr.w), r), ss = mul2(pk2(s.lzp.z, s.lzp.w), r);
      const u64 R = mul2(sz, r), Q = mul2(ss, r);
      w[0] = fma2(sz, d0, w[0]);
      w[1] = fma2(sz, d1, w[1]);
      w[2] = fma2(sz, d2, w[2]);
      w[3] = fma2(ss, d0, w[3]);
      w[4] = fma2(ss, d1, w[4]);
      w[5] = fma2(ss, d2, w[5]);
      const u64 r0 = mul2(R, d0), r1 = mul2(R, d1), r2 = mul2(R, d2);
      const u64 q0 = mul2(Q, d0), q1 = mul2(Q, d1), q2 = mul2(Q, d2);
      w[6] = add2(w[6], r0);
      w[7] = add2(w[7], r1);
      w[8] = add2(w[8], r2);
      w[9] = add2(w[9], q0);
      w[10] = add2(w[10], q1);
      w[11] = add2(w[11], q2);
      w[12] = fma2(r0, d0, w[12]);
      w[13] = fma2(r0, d1, w[13]);
      w[14] = fma2(r0, d2, w[14]);
      w[15] = fma2(r1, d1, w[15]);
      w[16] = fma2(r1, d2, w[16]);
      w[17] = fma2(r2, d2, w[17]);
      w[18] = fma2(q0, d0, w[18]);
      w[19] = fma2(q0, d1, w[19]);
      w[20] = fma2(q0, d2, w[20]);
      w[21] = fma2(q1, d1, w[21]);
      w[22] = fma2(q1, d2, w[22]);
      w[23] = fma2(q2, d2, w[23]);
      w[24] = add2(w[24], sz);
      w[25] = add2(w[25], ss);
      w[26] = fma2(ss, dd, w[26]);
    }
#pragma unroll
    for (int k = 0; k < kSph32NC; ++k) {
      float a, b;
      upk2(w[k], a, b);
      acc[k][tid] += double(a) + double(b);
    }
  }
  if (!valid) return;
#pragma unroll
  for (int k = 0; k < kSph32NC; ++k) part[(c * kSph32NC + k) * tpad + i] = acc[k][tid];
}

__global__ void k_swe_sphere32_out(const double* __restrict__ part, int64_t tpad, View tx, int64_t nt, double eps2, View u,
                                   double* __restrict__ ddot, double* __restrict__ grad,
                                   int do_velocity) {
  const int64_t i = blockIdx.x * int64_t(blockDim.x) + threadIdx.x;
  if (i >= nt) return;
  double s[kSph32NC];
#pragma unroll
  for (int k = 0; k < kSph32NC; ++k) s[k] = part[k * tpad + i];
  // the kernel's sz, ss were doubled (strengths stored as rot, pot / pi):
  // halve A, B, Z, G, H (exact)
  for (int k : {0, 1, 2, 3, 4, 5, 24, 25, 26}) s[k] *= 0.5;
  const double x[3] = {tx(i, 0), tx(i, 1), tx(i, 2)};
  const double *A = s, *B = s + 3, *U1 = s + 6, *V1 = s + 9;
  const int sym[9] = {0, 1, 2, 1, 3, 4, 2, 4, 5};  // (a, b) -> packed symmetric index
  const double *U2 = s + 12, *V2 = s + 18;
  const double Z = s[24], G = s[25], H = s[26];
  double P[9];
#pragma unroll
  for (int a = 0; a < 3; ++a)
#pragma unroll
    for (int b = 0; b < 3; ++b) P[3 * a + b] = (a == b ? 1.0 : 0.0) - x[a] * x[b];
  auto cross = [](const double* p, const double* q, double* o) {
    o[0] = p[1] * q[2] - p[2] * q[1];
    o[1] = p[2] * q[0] - p[0] * q[2];
    o[2] = p[0] * q[1] - p[1] * q[0];
  };
  if (do_velocity) {
    double ax[3];
    cross(A, x, ax);
#pragma unroll
    for (int a = 0; a < 3; ++a) u(i, a) = ax[a] - (P[3 * a] * B[0] + P[3 * a + 1] * B[1] + P[3 * a + 2] * B[2]);
  }
  double u1x[3], pv1[3], zy[3];
  cross(U1, x, u1x);
#pragma unroll
  for (int a = 0; a < 3; ++a) {
    pv1[a] = P[3 * a] * V1[0] + P[3 * a + 1] * V1[1] + P[3 * a + 2] * V1[2];
    zy[a] = Z * x[a] - A[a];
  }
  const double Yx[9] = {0.0, -zy[2], zy[1], zy[2], 0.0, -zy[0], -zy[1], zy[0], 0.0};
  const double g = G - 0.5 * H;
  double M[9];
#pragma unroll
  for (int b = 0; b < 3; ++b) {
    const double col[3] = {U2[sym[b]], U2[sym[3 + b]], U2[sym[6 + b]]};
    double t1[3];
    cross(col, x, t1);
#pragma unroll
    for (int a = 0; a < 3; ++a) {
      const double v2p = V2[sym[3 * a]] * P[b] + V2[sym[3 * a + 1]] * P[3 + b] + V2[sym[3 * a + 2]] * P[6 + b];
      M[3 * a + b] = eps2 * u1x[a] * x[b] + t1[a] + eps2 * x[a] * pv1[b] + v2p + Yx[3 * a + b] -
                     g * P[3 * a + b];
    }
  }
  double dsum = 0.0;
#pragma unroll
  for (int a = 0; a < 3; ++a)
#pragma unroll
    for (int b = 0; b < 3; ++b) dsum = da(dsum, dm(M[3 * a + b], M[3 * b + a]));
  ddot[i] = dsum;
  if (grad)
#pragma unroll
    for (int k = 0; k < 9; ++k) grad[9 * i + k] = M[k];
}

// The chunks' partials added in place (into the first chunk's), a thread per
// component and target: a thread per target reads 11 to 28 of them one chunk after
// the other, which on small grids took longer than the pair sums (and 0.25 of 2.9 ms
// at quad level 5).
__global__ void k_swe_sum(double* __restrict__ part, int nchunks, int64_t n) {
  const int64_t q = blockIdx.x * int64_t(blockDim.x) + threadIdx.x;
  if (q >= n) return;
  double s[1];
  sum_chunks<1>(part + q, nchunks, n, s);
  part[q] = s[0];
}

// Scratch and chunking shared by the four SWE paths: 128 targets per CTA,
// sources compacted (masked slots dropped) and split into chunks of whole
// tiles, about eight waves of CTAs; ncomp FP64 partials per (chunk, target),
// added in fixed order by the epilogue.
struct SwePlan {
  int64_t nb = 0, tpad = 0, ns = 0, chunk_len = 0;
  int nchunks = 1, threads = kSweNT;
  int* src2slot = nullptr;
  void* src = nullptr;     // ns packed source records
  int* slot = nullptr;     // ns slot indices (when asked for)
  double* tgt = nullptr;   // [tgt_doubles][tpad] (when asked for)
  double* part = nullptr;  // [chunk][ncomp][tpad]
  dim3 grid() const { return dim3{unsigned(nb), unsigned(nchunks), 1u}; }
};

SwePlan swe_plan(lpm_context& ctx, const uint8_t* mask, int64_t nt, int64_t nf, size_t rec_bytes,
                 int ncomp, bool want_slot, int tile, int tgt_doubles = 0) {
  SwePlan p;
  ctx.arena.reset();
  if (tile == kSweTile64) {
    // FP64: one warp's pair takes the FP64 pipe of its sub-partition 1,200 to 3,000
    // clocks, so few points are cut into chunks of down to 8 sources until every
    // sub-partition has two warps (quad level 2, vertices and faces, with the chunks'
    // sums by k_swe_sum: 306 -> 134 us); CTAs no larger than the targets.
    p.threads = int(std::min<int64_t>(kSweNT, (nt + 31) / 32 * 32));
    while (tile > 8 && (nt + 31) / 32 * ((nf + tile - 1) / tile) < int64_t(ctx.num_sms) * 8) tile /= 2;
  }
  p.nb = (nt + p.threads - 1) / p.threads;
  p.tpad = p.nb * p.threads;
  const int64_t want = std::max<int64_t>(1, (int64_t(ctx.num_sms) * 4 * 8 + p.nb - 1) / p.nb);
  const int64_t nch_max =
      std::max<int64_t>(1, std::min<int64_t>(want, (nf + tile - 1) / tile));
  ctx.arena.reserve(sizeof(int) * (3 * size_t(nf) + 2 * size_t(nf) / 1024 + 8) +
                    rec_bytes * size_t(nf) +
                    sizeof(double) * (ncomp * size_t(nch_max) + tgt_doubles) * p.tpad +
                    8 * 4096);
  int* slot2src = static_cast<int*>(ctx.arena.take(sizeof(int) * std::max<int64_t>(nf, 1)));
  p.src2slot = static_cast<int*>(ctx.arena.take(sizeof(int) * std::max<int64_t>(nf, 1)));
  p.ns = compact_sources(ctx, mask, nf, slot2src, p.src2slot);
  // one record more than the sources: the FP32 spherical path packs pairs
  p.src = ctx.arena.take(rec_bytes * size_t(p.ns + 1));
  if (want_slot) p.slot = static_cast<int*>(ctx.arena.take(sizeof(int) * size_t(p.ns + 1)));
  int64_t len = (p.ns + nch_max - 1) / nch_max;
  p.chunk_len = std::max<int64_t>(tile, (len + tile - 1) / tile * tile);
  p.nchunks = int(std::max<int64_t>(1, (p.ns + p.chunk_len - 1) / p.chunk_len));
  if (tgt_doubles) p.tgt = static_cast<double*>(ctx.arena.take(sizeof(double) * tgt_doubles * p.tpad));
  p.part = static_cast<double*>(ctx.arena.take(sizeof(double) * ncomp * size_t(p.nchunks) * p.tpad));
  return p;
}

unsigned blocks256(int64_t n) { return unsigned((n + 255) / 256); }

void swe_sum(lpm_context& ctx, const SwePlan& p, int ncomp) {
  if (p.nchunks == 1) return;
  const int64_t n = ncomp * p.tpad;
  k_swe_sum<<<blocks256(n), 256, 0, ctx.stream>>>(p.part, p.nchunks, n);
  ctx.launches++;
}

void swe_sphere_sums32(lpm_context& ctx, View tx, int64_t nt, View fx, const double* zeta,
                       const double* sigma, const double* area, const uint8_t* mask, int64_t nf,
                       double eps, bool collocated, View u, double* ddot, double* grad,
                       int do_velocity) {
  // one 64-byte pair record per two sources (32 bytes per source, plus one
  // dummy for an odd count); the pair slots take the plan's slot array
  const SwePlan p = swe_plan(ctx, mask, nt, nf, sizeof(SphPair32) / 2, kSph32NC, true, kSweTile);
  auto* src = static_cast<SphPair32*>(p.src);
  auto* pslot = reinterpret_cast<int2*>(p.slot);
  if (p.ns > 0) {
    k_swe_sphere32_pack<<<blocks256((p.ns + 1) / 2), 256, 0, ctx.stream>>>(
        fx, zeta, sigma, area, p.src2slot, p.ns, src, pslot);
    ctx.launches++;
  }
  const float c0 = float(2 * eps * eps);
  if (collocated)
    k_swe_sphere32<true><<<p.grid(), kSweNT, 0, ctx.stream>>>(tx, nt, src, pslot, p.ns,
                                                              p.chunk_len, c0, p.part, p.tpad);
  else
    k_swe_sphere32<false><<<p.grid(), kSweNT, 0, ctx.stream>>>(tx, nt, src, pslot, p.ns,
                                                               p.chunk_len, c0, p.part, p.tpad);
  swe_sum(ctx, p, kSph32NC);
  k_swe_sphere32_out<<<blocks256(nt), 256, 0, ctx.stream>>>(p.part, p.tpad, tx, nt,
                                                            eps * eps, u, ddot, grad, do_velocity);
  ctx.launches += 2;
  LPM_CUDA(cudaGetLastError());
}

// Targets tx (nt x 3); sources: face slots fx/zeta/sigma/area/mask (nf);
// collocated: targets are the face slots themselves (i == j skipped).
void swe_sphere_sums(lpm_context& ctx, View tx, int64_t nt, View fx, const double* zeta,
                     const double* sigma, const double* area, const uint8_t* mask, int64_t nf,
                     double eps, bool collocated, View u, double* ddot, double* grad,
                     int do_velocity) {
  if (nt == 0) return;
  if (ctx.precision == LPM_FP32C) {
    swe_sphere_sums32(ctx, tx, nt, fx, zeta, sigma, area, mask, nf, eps, collocated, u, ddot, grad,
                      do_velocity);
    return;
  }
  const SwePlan p = swe_plan(ctx, mask, nt, nf, sizeof(SphSrc), kSphNC, false, kSweTile64, kSphFrame);
  auto* src = static_cast<SphSrc*>(p.src);
  const unsigned nblk = unsigned((p.ns + 127) / 128 + (nt + 127) / 128);
  k_swe_sphere_pack<<<nblk, 128, 0, ctx.stream>>>(fx, zeta, sigma, area, p.src2slot, p.ns, src, tx,
                                                  nt, p.tpad, p.tgt);
  ctx.launches++;
  if (collocated)
    k_swe_sphere<true><<<p.grid(), p.threads, 0, ctx.stream>>>(tx, nt, p.tgt, src, p.ns, p.chunk_len,
                                                               eps * eps, p.part, p.tpad);
  else
    k_swe_sphere<false><<<p.grid(), p.threads, 0, ctx.stream>>>(tx, nt, p.tgt, src, p.ns, p.chunk_len,
                                                                eps * eps, p.part, p.tpad);
  swe_sum(ctx, p, kSphNC);
  const unsigned th = unsigned(sum_threads(nt));
  k_swe_sphere_out<<<unsigned((nt + th - 1) / th), th, 0, ctx.stream>>>(
      p.part, p.tpad, p.tgt, nt, u, ddot, grad, do_velocity);
  ctx.launches += 2;
  LPM_CUDA(cudaGetLastError());
}

bool bad_count(int64_t n) { return n < 0 || n > (int64_t(1) << 31) - 1; }

// FloatingPoint<Real>::zero (src/util/lpm_floating_point.hpp:26-29): |x| < DBL_EPSILON
bool fp_zero(double x) { return std::fabs(x) < 2.220446049250313e-16; }

// Targets tx (nt x 2) with surface ts; sources: face slots fx/zeta/sigma/
// area/mask/sfc (nf); collocated: targets are the face slots themselves.
void swe_plane_sums32(lpm_context& ctx, View tx, const double* ts, int64_t nt, View fx,
                      const double* zeta, const double* sigma, const double* area,
                      const uint8_t* mask, const double* sfc, int64_t nf, double eps,
                      double pse_eps, bool collocated, const SweOut& out) {
  // one 80-byte pair record per two sources (plus one dummy for an odd count)
  const SwePlan p = swe_plan(ctx, mask, nt, nf, sizeof(PlPair32) / 2, kPl32NC, false, kSweTile);
  auto* src = static_cast<PlPair32*>(p.src);
  if (p.ns > 0) {
    k_swe_plane32_pack<<<blocks256((p.ns + 1) / 2), 256, 0, ctx.stream>>>(
        fx, zeta, sigma, area, sfc, p.src2slot, p.ns, src);
    ctx.launches++;
  }
  const float e2 = float(eps * eps), ipse2 = float(1.0 / (pse_eps * pse_eps));
  if (collocated)
    k_swe_plane32<true><<<p.grid(), kSweNT, 0, ctx.stream>>>(tx, ts, nt, src, p.ns, p.chunk_len,
                                                             e2, ipse2, p.part, p.tpad);
  else
    k_swe_plane32<false><<<p.grid(), kSweNT, 0, ctx.stream>>>(tx, ts, nt, src, p.ns, p.chunk_len,
                                                              e2, ipse2, p.part, p.tpad);
  swe_sum(ctx, p, kPl32NC);
  k_swe_plane32_out<<<blocks256(nt), 256, 0, ctx.stream>>>(p.part, p.tpad, nt, pse_eps,
                                                           out);
  ctx.launches += 2;
  LPM_CUDA(cudaGetLastError());
}

void swe_plane_sums(lpm_context& ctx, View tx, const double* ts, int64_t nt, View fx,
                    const double* zeta, const double* sigma, const double* area,
                    const uint8_t* mask, const double* sfc, int64_t nf, double eps,
                    double pse_eps, bool collocated, const SweOut& out) {
  if (nt == 0) return;
  if (ctx.precision == LPM_FP32C) {
    swe_plane_sums32(ctx, tx, ts, nt, fx, zeta, sigma, area, mask, sfc, nf, eps, pse_eps,
                     collocated, out);
    return;
  }
  const SwePlan p = swe_plan(ctx, mask, nt, nf, sizeof(SweSrc), kSweNC, false, kSweTile64);
  auto* src = static_cast<SweSrc*>(p.src);
  if (p.ns > 0) {
    k_swe_pack<<<blocks256(p.ns), 256, 0, ctx.stream>>>(fx, zeta, sigma, area, sfc, p.src2slot, p.ns,
                                                        src);
    ctx.launches++;
  }
  const double epssq = eps * eps, ipse2 = 1.0 / (pse_eps * pse_eps);
  if (collocated)
    k_swe_plane<true><<<p.grid(), p.threads, 0, ctx.stream>>>(tx, ts, nt, src, p.ns, p.chunk_len, epssq,
                                                           ipse2, ctx.f64_tab, p.part, p.tpad);
  else
    k_swe_plane<false><<<p.grid(), p.threads, 0, ctx.stream>>>(tx, ts, nt, src, p.ns, p.chunk_len,
                                                            epssq, ipse2, ctx.f64_tab, p.part, p.tpad);
  swe_sum(ctx, p, kSweNC);
  const unsigned th = unsigned(sum_threads(nt));
  k_swe_out<<<unsigned((nt + th - 1) / th), th, 0, ctx.stream>>>(p.part, p.tpad, nt, pse_eps, out);
  ctx.launches += 2;
  LPM_CUDA(cudaGetLastError());
}

}  // namespace
}  // namespace lpm

namespace {
int swe_args(lpm_context* ctx, lpm_view u, double* ddot, double* a, double* b, double* c,
             double* d, double* laps, double* psi, double* phi, lpm_view x, const double* s,
             int64_t nt, lpm_view fx, const double* zeta, const double* sigma, const double* area,
             const uint8_t* mask, const double* fs, int64_t nf, double eps, double pse_eps,
             int do_velocity) {
  if (!ctx) return lpm::fail(LPM_ERR_ARG, "null context");
  if (lpm::bad_count(nt) || lpm::bad_count(nf))
    return lpm::fail(LPM_ERR_ARG, "count out of range [0, 2^31-1]");
  if (nt > 0 && (!x.p || !s || !ddot || !a || !b || !c || !d || !laps || !psi || !phi ||
                 (do_velocity && !u.p)))
    return lpm::fail(LPM_ERR_ARG, "null target or output array");
  if (nf > 0 && (!fx.p || !zeta || !sigma || !area || !mask || !fs))
    return lpm::fail(LPM_ERR_ARG, "null source array");
  if (!(eps >= 0) || !std::isfinite(eps) || !(pse_eps > 0) || !std::isfinite(pse_eps))
    return lpm::fail(LPM_ERR_ARG, "eps must be >= 0 and pse_eps > 0, both finite");
  return LPM_OK;
}
}  // namespace

extern "C" {

int lpm_swe_plane_vertex_sums(lpm_context* ctx, lpm_view u, double* ddot, double* du1dx1,
                              double* du1dx2, double* du2dx1, double* du2dx2, double* laps,
                              double* psi, double* phi, lpm_view vx, const double* vs, int64_t nv,
                              lpm_view fx, const double* fzeta, const double* fsigma,
                              const double* farea, const uint8_t* fmask, const double* fs,
                              int64_t nf, double eps, double pse_eps, int do_velocity) {
  if (int r = swe_args(ctx, u, ddot, du1dx1, du1dx2, du2dx1, du2dx2, laps, psi, phi, vx, vs, nv,
                       fx, fzeta, fsigma, farea, fmask, fs, nf, eps, pse_eps, do_velocity))
    return r;
  try {
    lpm::DeviceGuard device_guard(ctx->device);
    lpm::SweOut o{lpm::to_view(u), ddot, du1dx1, du1dx2, du2dx1, du2dx2, laps, psi, phi, do_velocity};
    lpm::swe_plane_sums(*ctx, lpm::to_view(vx), vs, nv, lpm::to_view(fx), fzeta, fsigma, farea,
                        fmask, fs, nf, eps, pse_eps, false, o);
    return LPM_OK;
  } catch (...) {
    return lpm::handle_exception();
  }
}

int lpm_swe_plane_face_sums(lpm_context* ctx, lpm_view u, double* ddot, double* du1dx1,
                            double* du1dx2, double* du2dx1, double* du2dx2, double* laps,
                            double* psi, double* phi, lpm_view fx, const double* fzeta,
                            const double* fsigma, const double* farea, const uint8_t* fmask,
                            const double* fs, int64_t nf, double eps, double pse_eps,
                            int do_velocity) {
  if (int r = swe_args(ctx, u, ddot, du1dx1, du1dx2, du2dx1, du2dx2, laps, psi, phi, fx, fs, nf,
                       fx, fzeta, fsigma, farea, fmask, fs, nf, eps, pse_eps, do_velocity))
    return r;
  try {
    lpm::DeviceGuard device_guard(ctx->device);
    lpm::SweOut o{lpm::to_view(u), ddot, du1dx1, du1dx2, du2dx1, du2dx2, laps, psi, phi, do_velocity};
    // PlanarSWEFaceSums: collocated = FloatingPoint<Real>::zero(eps)
    lpm::swe_plane_sums(*ctx, lpm::to_view(fx), fs, nf, lpm::to_view(fx), fzeta, fsigma, farea,
                        fmask, fs, nf, eps, pse_eps, lpm::fp_zero(eps), o);
    return LPM_OK;
  } catch (...) {
    return lpm::handle_exception();
  }
}

int lpm_swe_sphere_vertex_sums(lpm_context* ctx, lpm_view u, double* ddot, double* grad,
                               lpm_view vx, int64_t nv, lpm_view fx, const double* fzeta,
                               const double* fsigma, const double* farea, const uint8_t* fmask,
                               int64_t nf, double eps, int do_velocity) {
  if (!ctx) return lpm::fail(LPM_ERR_ARG, "null context");
  if (lpm::bad_count(nv) || lpm::bad_count(nf))
    return lpm::fail(LPM_ERR_ARG, "count out of range [0, 2^31-1]");
  if (nv > 0 && (!vx.p || !ddot || (do_velocity && !u.p)))
    return lpm::fail(LPM_ERR_ARG, "null target or output array");
  if (nf > 0 && (!fx.p || !fzeta || !fsigma || !farea || !fmask))
    return lpm::fail(LPM_ERR_ARG, "null source array");
  if (!(eps >= 0) || !std::isfinite(eps)) return lpm::fail(LPM_ERR_ARG, "eps must be finite and >= 0");
  try {
    lpm::DeviceGuard device_guard(ctx->device);
    lpm::swe_sphere_sums(*ctx, lpm::to_view(vx), nv, lpm::to_view(fx), fzeta, fsigma, farea, fmask,
                         nf, eps, false, lpm::to_view(u), ddot, grad, do_velocity);
    return LPM_OK;
  } catch (...) {
    return lpm::handle_exception();
  }
}

int lpm_swe_sphere_face_sums(lpm_context* ctx, lpm_view u, double* ddot, double* grad,
                             lpm_view fx, const double* fzeta, const double* fsigma,
                             const double* farea, const uint8_t* fmask, int64_t nf, double eps,
                             int do_velocity) {
  if (!ctx) return lpm::fail(LPM_ERR_ARG, "null context");
  if (lpm::bad_count(nf)) return lpm::fail(LPM_ERR_ARG, "count out of range [0, 2^31-1]");
  if (nf > 0 && (!fx.p || !fzeta || !fsigma || !farea || !fmask || !ddot || (do_velocity && !u.p)))
    return lpm::fail(LPM_ERR_ARG, "null input or output array");
  if (!(eps >= 0) || !std::isfinite(eps)) return lpm::fail(LPM_ERR_ARG, "eps must be finite and >= 0");
  try {
    lpm::DeviceGuard device_guard(ctx->device);
    // SphereFaceSums: collocated = FloatingPoint<Real>::zero(eps)
    lpm::swe_sphere_sums(*ctx, lpm::to_view(fx), nf, lpm::to_view(fx), fzeta, fsigma, farea, fmask,
                         nf, eps, lpm::fp_zero(eps), lpm::to_view(u), ddot, grad, do_velocity);
    return LPM_OK;
  } catch (...) {
    return lpm::handle_exception();
  }
}

}  // extern "C"
