// f64math.cuh -- FP64 logarithm, exponential and reciprocal for pair loops that
// the FP64 pipe bounds (about 1.7 operations per clock per SM): table lookups and
// integer operations, which run beside it, take the place of FP64 ones.
//
// log x: x = 2^k m; f = 1/c for the centre c of m's interval of width 2^-9 (table),
// r = m f - 1 (fused), log x = k ln 2 - log f + log1p(r), the series to r^5 / 5 for
// |r| <= 2^-10: 9 FP64 operations.
// exp(-p): -p = (256 n + j) ln 2 / 256 + f, 2^(j/256) from a table, exp(f) by its
// series to f^5 / 120 for |f| <= ln 2 / 512: 11 FP64 operations.
// Both from the textbook reductions (Cody and Waite; Tang's table-driven
// methods); absolute error of log about 2e-16 (1 + |log x| / 2), relative error of
// exp about 3e-16.
#pragma once

#include <cuda_runtime.h>

namespace lpm {

constexpr int kLogBits = 9;
struct F64Tables {
  double2 lg[1 << kLogBits];  // f, -log f (less ln 2 above sqrt 2)
  double ex[256];             // 2^(j/256)
};
constexpr double kLn2 = 0.69314718055994530942;

constexpr double kMagic = 6755399441055744.0;  // 2^52 + 2^51: integers in the low word

// Entry i of the tables, i in [0, 2^kLogBits).
__device__ __forceinline__ void f64_table_entry(F64Tables* T, int i) {
  {
    const double c = 1.0 + (i + 0.5) / (1 << kLogBits);
    const double f = 1.0 / c;
    T->lg[i] = make_double2(f, -log(f) - (c > 1.41421356237309504880 ? kLn2 : 0.0));
  }
  if (i < 256) T->ex[i] = exp2(i / 256.0);
}

// Whether x is a positive normal number in [2^-1000, 2^1000).
__device__ __forceinline__ bool f64_plain(double x) {
  const unsigned h = unsigned(__double2hiint(x));
  return h - (23u << 20) < (2000u << 20);
}

// 1/d, d as f64_plain: the approximate reciprocal (relative error e below
// 2^-20) times 1 + e + e^2.
__device__ __forceinline__ double f64_rcp(double d) {
  double r;
  asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(r) : "d"(d));
  const double e = fma(-d, r, 1.0);
  return fma(r, fma(e, e, e), r);
}

__device__ __forceinline__ double f64_log(const F64Tables& T, double x) {
  const int h = __double2hiint(x);
  const int i = (h >> (20 - kLogBits)) & ((1 << kLogBits) - 1);
  const double2 t = T.lg[i];
  // above sqrt 2 the table holds -log f - ln 2 and the exponent counts one more
  const int k = (h >> 20) - 1023 + (t.y < 0.0 ? 1 : 0);
  const double m = __hiloint2double((h & 0xfffff) | 0x3ff00000, __double2loint(x));
  const double kd = __hiloint2double(0x43380000, k + 2048) - (kMagic + 2048.0);
  const double r = fma(m, t.x, -1.0);
  double p = fma(r, 0.2, -0.25);
  p = fma(r, p, 1.0 / 3);
  p = fma(r, p, -0.5);
  return fma(kd, kLn2, t.y) + fma(r * r, p, r);
}

// q exp(-p) for 0 <= p < 746 (beyond, exp(-p) is 0 in FP64); q finite.
__device__ __forceinline__ double f64_mul_exp_neg(const F64Tables& T, double q, double p) {
  const double z = fma(p, -369.3299304675746, kMagic);  // -256 / ln 2
  const int n = __double2loint(z);
  const double zf = z - kMagic;
  // ln 2 / 256 in two parts, the first of 29 bits: zf times it is exact
  double f = fma(zf, -0x1.62e42fep-9, -p);
  f = fma(zf, -0x1.f473de6af278fp-38, f);
  double e = fma(f, 1.0 / 120, 1.0 / 24);
  e = fma(f, e, 1.0 / 6);
  e = fma(f, e, 0.5);
  e = fma(f * f, e, f);
  // 2^k into the exponent of the table value, as far as it stays normal
  const double t0 = T.ex[n & 255];
  const int k = n >> 8, k1 = max(k, -1000);
  const double t = __hiloint2double(__double2hiint(t0) + (k1 << 20), __double2loint(t0));
  double v = q * fma(t, e, t);
  if (k < k1) v *= __hiloint2double((1023 + k - k1) << 20, 0);
  return v;
}

}  // namespace lpm
