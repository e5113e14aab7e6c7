// f64math.cuh -- FP64 logarithm, exponential and reciprocal for pair loops that
// the FP64 pipe bounds (about 1.7 operations per clock per SM: 64 clocks of a
// sub-partition's pipe per warp instruction).  The other pipes' issue slots are
// free there, so the values are formed in 64-bit fixed point (integer operations,
// FP32 for the last terms) and tables, and rounded to FP64 once:
//
// 1/x: FP32 reciprocal y of the mantissa m, e = 1 - m y exactly (integers modulo
// 2^64), y (1 + e + e^2): no FP64 operation.
// log x: x = 2^k m; f = 1/c to 22 bits for the centre c of m's interval of width
// 2^-12 (table), r = m f - 1 exactly (integers modulo 2^64), log x = (k ln 2 - log f)
// + log1p(r), the series to r^5 / 5 in fixed point of 74 bits: 2 FP64 additions.
// exp(-p): p = n ln 2 / 8192 + r in fixed point of 76 bits, 2^(-n/8192) from a table of
// 63 bits, exp(-r) by its series to r^4 / 24; the polynomial before it in 61 bits: no
// FP64 operation.
// The range reductions are those of Cody and Waite, and Tang's table-driven
// methods.  Errors: 1/x and exp about half a unit in the last place, log
// two roundings of its parts.  The tables (145 KB) are read through L1.
#pragma once

#include <cstdint>

#include <cuda_runtime.h>

namespace lpm {

constexpr int kLogBits = 12, kExpBits = 13;
constexpr int kF64Entries = 1 << kExpBits;  // of the largest table
constexpr double kLn2 = 0.69314718055994530942;
struct __align__(16) F64LogEntry {
  double y;    // -log f, less ln 2 above sqrt 2
  unsigned f;  // 2^22 f
  unsigned up;  // 1 above sqrt 2: the exponent counts one more
};
struct __align__(16) F64Tables {
  F64LogEntry lg[1 << kLogBits];
  uint64_t ex[1 << kExpBits];  // 2^63 2^(-j / 2^kExpBits)
  double kl[2050];             // (e - 1023) ln 2
};

// Entry i of the tables, i in [0, kF64Entries).
__device__ __forceinline__ void f64_table_entry(F64Tables* T, int i) {
  if (i < 1 << kLogBits) {
    // f = 1 beside 1 and 1/2 beside 2: log x stays accurate relative to x - 1
    const double c = i == 0 ? 1.0 : i == (1 << kLogBits) - 1 ? 2.0 : 1.0 + (i + 0.5) / (1 << kLogBits);
    const unsigned f = unsigned(rint(0x1p22 / c));
    const bool up = c > 1.41421356237309504880;
    T->lg[i] = F64LogEntry{-log(f * (up ? 0x1p-21 : 0x1p-22)), f, unsigned(up)};
  }
  if (i < 2050) T->kl[i] = (i - 1023) * kLn2;
  // 2^64 2^(-2^k / 8192), multiplied over the bits of i
  constexpr uint64_t root[kExpBits] = {
      0xfffa747ea0040664ull, 0xfff4e91bff1b8c3eull, 0xffe9d2b2f7db2756ull, 0xffd3a751c0f7e10cull,
      0xffa756521c8daed2ull, 0xff4ecb59511ec8a5ull, 0xfe9e115c7b8f884cull, 0xfd3e0c0cf486c175ull,
      0xfa83b2db722a033aull, 0xf5257d152486cc2cull, 0xeac0c6e7dd24392full, 0xd744fccad69d6af4ull,
      0xb504f333f9de6484ull};
  uint64_t t = uint64_t(1) << 63;
#pragma unroll
  for (int k = 0; k < kExpBits; ++k)
    if (i >> k & 1) t = __umul64hi(t, root[k]);
  T->ex[i] = t;
}

// A float as a double by its bits: the conversion instruction holds the FP64 pipe as
// long as an addition.
static __device__ __noinline__ double f64_widen_any(float v) { return double(v); }
__device__ __forceinline__ double f64_widen(float v) {
  const unsigned b = __float_as_uint(v), m = b & 0x7fffffffu;
  if (m - 0x00800000u < 0x7f000000u)  // normal
    return __hiloint2double(int((b & 0x80000000u) | ((m >> 3) + (896u << 20))), int(b << 29));
  return m == 0 ? 0.0 : f64_widen_any(v);
}

// Whether x is a positive normal number in [2^-1000, 2^1000).
__device__ __forceinline__ bool f64_plain(double x) {
  const unsigned h = unsigned(__double2hiint(x));
  return h - (23u << 20) < (2000u << 20);
}

__device__ __forceinline__ uint64_t f64_mantissa(double x) {  // 2^52 m, m in [1, 2)
  return (uint64_t(__double_as_longlong(x)) & 0xfffffffffffffull) | 0x10000000000000ull;
}
// a 2^(e - 1086) rounded to nearest, for the normalised a (bit 63 set) and the biased
// exponent e of the result
__device__ __forceinline__ uint64_t f64_pack(uint64_t a, int e) {
  return (a >> 11) + (a >> 10 & 1) + (uint64_t(unsigned(e - 1)) << 52);
}

// -1^neg mag 2^k, within the normal range.
__device__ __forceinline__ double f64_value(uint64_t mag, bool neg, int k) {
  const int z = __clzll(int64_t(mag | 1));
  const uint64_t b = mag != 0 ? f64_pack(mag << z, 1086 - z + k) : 0;
  return __hiloint2double(int(unsigned(b >> 32) | (neg ? 0x80000000u : 0u)), int(unsigned(b)));
}

// 2^63 / m for the mantissa m of d.
__device__ __forceinline__ uint64_t f64_rcp_mantissa(double d) {
  const unsigned h = unsigned(__double2hiint(d)), l = unsigned(__double2loint(d));
  const float mh = __int_as_float(int(__funnelshift_l(l, h & 0xfffff, 3)) | 0x3f800000);
  float y;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(mh));
  y = fminf(y, 0x1.fffffep-1f);
  const unsigned Y = (unsigned(__float_as_int(y)) & 0x7fffff) | 0x800000;  // 2^24 y
  const int64_t E = -int64_t(f64_mantissa(d) * Y);                         // 2^76 (1 - m y)
  const int e = int(E >> 32);                                              // 2^44 e
  const int64_t e2 = (int64_t(e) * e) >> 24;                               // 2^64 e^2
  return (uint64_t(Y) << 39) + uint64_t((int64_t(Y) * (E >> 16)) >> 21) +
         ((uint64_t(unsigned(e2)) * Y) >> 25);
}
// The reciprocal with that mantissa.
__device__ __forceinline__ double f64_rcp_value(uint64_t W, double d) {
  const unsigned h = unsigned(__double2hiint(d));
  const uint64_t b = ((W + 0x200) >> 10) + (uint64_t(2044 - ((h >> 20) & 0x7ff)) << 52);
  return __hiloint2double(int(unsigned(b >> 32) | (h & 0x80000000u)), int(unsigned(b)));
}
// 1/d, |d| as f64_plain.
__device__ __forceinline__ double f64_rcp(double d) {
  return f64_rcp_value(f64_rcp_mantissa(d), d);
}
// 1/d for any d.  The rare case is a call: inlined, its FP64 operations are issued
// for every pair and the result selected.
static __device__ __noinline__ double f64_inv_any(double d) { return 1.0 / d; }
__device__ __forceinline__ double f64_inv(double d) {
  return f64_plain(fabs(d)) ? f64_rcp(d) : f64_inv_any(d);
}

// log x, x as f64_plain and not within 2^-16 of 1 (where the error, 2^-67, outgrows
// the result's last place).
__device__ __forceinline__ double f64_log(const F64Tables* __restrict__ T, double x) {
  const int h = __double2hiint(x);
  const int4 t4 = reinterpret_cast<const int4*>(T->lg)[(h >> (20 - kLogBits)) & ((1 << kLogBits) - 1)];
  const double base = T->kl[(h >> 20) + t4.w] + __hiloint2double(t4.y, t4.x);
  const int64_t r = int64_t(f64_mantissa(x) * unsigned(t4.z));  // 2^74 r, |r| < 2^-12
  const float rf = float(int(r >> 32)) * 0x1p-42f;
  const int c = __float2int_rn(rf * rf * rf * fmaf(rf, fmaf(rf, 0.2f, -0.25f), 1.f / 3) * 0x1p66f);
  const int64_t v = r - (__mul64hi(r << 1, r << 1) >> 13) + (int64_t(c) << 8);  // 2^74 log1p(r)
  const uint64_t a = uint64_t(v < 0 ? -v : v);
  const int z = __clzll(int64_t(a | 1));
  const uint64_t b = ((a << z) >> 11) + (uint64_t(unsigned(1023 - 12 - z)) << 52);
  return base + __hiloint2double(int(unsigned(b >> 32) | (unsigned(v >> 32) & 0x80000000u)),
                                 int(unsigned(b)));
}
// Whether x is one that f64_log takes.
__device__ __forceinline__ bool f64_log_plain(double x) {
  return f64_plain(x) && unsigned(__double2hiint(x)) - 0x3fefffe0u >= 0x30u;
}
// log x for any x.
static __device__ __noinline__ double f64_ln_any(double x) { return log(x); }
__device__ __forceinline__ double f64_ln(const F64Tables* __restrict__ T, double x) {
  return f64_log_plain(x) ? f64_log(T, x) : f64_ln_any(x);
}

// (40 (1 - p) + 10 p^2 - 2 p^3 / 3) exp(-p) for p = m 2^(ep - 63), m in [2^63, 2^64),
// p < 746 (beyond, exp(-p) is 0 in FP64).  The cubic by Horner's rule in f = p / 2^K
// < 1, K >= 3, times 2^-3K, in 61 bits.
__device__ __forceinline__ double f64_pse8(const F64Tables* __restrict__ T, uint64_t m, int ep) {
  const uint64_t P = m >> min(9 - ep, 63);  // 2^54 p
  const unsigned n = unsigned((uint64_t(unsigned(P >> 32)) * 12102203u) >> 32);
  const int64_t r = int64_t((P << 22) - n * 0x58b90bfbe8e7bcd6ull);  // 2^76 r, r < 2^-13.4
  const int r1 = int((r + (int64_t(1) << 31)) >> 32);                // 2^44 r
  const float rf = float(r1) * 0x1p-44f;
  const int c = __float2int_rn(rf * rf * rf * fmaf(rf, -1.f / 24, 1.f / 6) * 0x1p70f);
  const int64_t v = ((int64_t(r1) * r1) >> 13) - r - (int64_t(c) << 6);  // 2^76 (exp(-r) - 1)
  const uint64_t t = T->ex[n & ((1 << kExpBits) - 1)];
  const uint64_t E = t + uint64_t(__mul64hi(int64_t(t >> 1), v) >> 11);  // 2^63 2^(-j/8192 - r)

  const int K = max(ep + 1, 3);
  const int64_t f = int64_t(m >> min(K - ep, 63));  // 2^63 p / 2^K
  constexpr int64_t k5 = int64_t(5) << 60;          // 40 in 2^61, over 2^4
  int64_t g = (k5 >> (K - 2)) - __mul64hi(0x2aaaaaaaaaaaaaabll, f);
  g = 2 * __mul64hi(g, f) - (k5 >> (2 * K - 4));
  g = 2 * __mul64hi(g, f) + (k5 >> (3 * K - 4));

  // 2^61 |g| 2^(-j/8192 - r); E = 2^63 less one
  const uint64_t h = __umul64hi(uint64_t(g < 0 ? -g : g), (E - (E >> 63)) << 1);
  const int z = __clzll(int64_t(h | 1));
  const int e = 1023 + 2 - z + 3 * K - int(n >> kExpBits), e1 = max(e, 23);
  const uint64_t b = f64_pack(h << z, e1);
  double w = __hiloint2double(int(unsigned(b >> 32) | (unsigned(g >> 32) & 0x80000000u)),
                              int(unsigned(b)));
  if (e < e1) w *= __hiloint2double((1023 + e - e1) << 20, 0);
  return w;
}

}  // namespace lpm
