// exact_f64.cuh -- IEEE double division, square root and a few other double
// operations on the 32-bit integer pipes, rounded to nearest even like the
// operations they replace, bit for bit.
//
// GB300 issues two double-precision results a cycle per SM; a correctly rounded
// quotient or root made of such operations takes ten or so of them, and a
// Hydro step forms sixty per cell: 2.62 ms for a 1024^2 step, all of it on that
// pipe (1.17 ms with these).  The integer pipes do 64 operations a cycle.  Here a quotient is two
// integer digits of about 30 and 25 bits, each from a 32-bit fixed-point
// reciprocal (a single-precision seed and one Newton step), with the remainder
// kept exactly; the last remainder decides the rounding.  That is schoolbook
// division with an estimated digit (Knuth, The Art of Computer Programming
// vol. 2, 4.3.1) in base 2^30; the root is the same digit by digit with the
// remainder x - s^2.
//
// The code is plain C++ besides the seeds, so that it runs on the host too.
#pragma once

#include <stdint.h>
#include <string.h>

#ifdef __CUDACC__
#include <cuda_runtime.h>
#define XF_FN __host__ __device__ __forceinline__
#define XF_SLOW static __host__ __device__ __noinline__
#else
#include <cmath>
#define XF_FN inline
#define XF_SLOW static inline
#endif

namespace om {
namespace xf {

XF_FN uint64_t bits(double x) {
#ifdef __CUDA_ARCH__
  return (uint64_t)__double_as_longlong(x);
#else
  uint64_t u;
  memcpy(&u, &x, 8);
  return u;
#endif
}
XF_FN double from_bits(uint64_t u) {
#ifdef __CUDA_ARCH__
  return __longlong_as_double((long long)u);
#else
  double x;
  memcpy(&x, &u, 8);
  return x;
#endif
}
XF_FN uint32_t hi32(uint64_t u) { return (uint32_t)(u >> 32); }
XF_FN uint32_t mulhi(uint32_t a, uint32_t b) { return (uint32_t)(((uint64_t)a * b) >> 32); }
// d * b mod 2^64 for a 32-bit digit d
XF_FN uint64_t mul_digit(uint32_t d, uint64_t b) {
  return (uint64_t)d * (uint32_t)b + ((uint64_t)(d * hi32(b)) << 32);
}
XF_FN float float_bits(uint32_t u) {
#ifdef __CUDA_ARCH__
  return __uint_as_float(u);
#else
  float f;
  memcpy(&f, &u, 4);
  return f;
#endif
}
XF_FN uint32_t bits_float(float f) {
#ifdef __CUDA_ARCH__
  return __float_as_uint(f);
#else
  uint32_t u;
  memcpy(&u, &f, 4);
  return u;
#endif
}

// Seeds: 1 / f and 1 / sqrt(f) within a few units of the 23rd bit.  XF_SEED
// lets a host test disturb them.
#ifndef XF_SEED
#define XF_SEED(y) (y)
#endif
XF_FN float seed_rcp(float f) {
#ifdef __CUDA_ARCH__
  float y;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(f));
  return y;
#else
  return XF_SEED(1.0f / f);
#endif
}
XF_FN float seed_rsqrt(float f) {
#ifdef __CUDA_ARCH__
  float y;
  asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(f));
  return y;
#else
  return XF_SEED(1.0f / std::sqrt(f));
#endif
}

// (1/2, which is below both 1 / f for f < 2 and 1 / sqrt(f) for f < 4)
XF_FN float at_least_half(float y) { return y < 0.5f ? 0.5f : y; }

// Operands whose exponents lie in [kLo, kHi) divide, take roots and halve with
// normal results; others take the plain operation.
constexpr uint32_t kLo = (1023u - 480u) << 20, kSpan = 960u << 20;
XF_FN bool plain_exponent(uint32_t h) { return (h & 0x7fffffffu) - kLo < kSpan; }

// A divisor with its 32-bit reciprocal.
struct Divisor {
  double b;
  uint64_t m;    // mantissa, in [2^52, 2^53)
  uint32_t y;    // 2^32 / (m / 2^52), from below, within 2^-28.4 of it
  uint32_t h;    // upper word of b
};

XF_FN Divisor divisor(double b) {
  Divisor d;
  const uint64_t u = bits(b);
  d.b = b;
  d.h = hi32(u);
  d.m = (u & 0x000fffffffffffffull) | 0x0010000000000000ull;
  // f = the upper 24 mantissa bits, f <= m / 2^52 < f (1 + 2^-23); the seed of
  // 1 / f is lowered by 2^-20.4 to be below 1 / (m / 2^52) whatever its error
  // (a few units of 2^-23), and below 1
  const float f = float_bits((uint32_t)(d.m >> 29) + 0x3f000000u);
  float y = seed_rcp(f);
  y = at_least_half(y - y * 7.2e-7f);
  const uint32_t y0 = (bits_float(y) << 8) | 0x80000000u;
  // Newton: t / 2^31 = 1 - y m at most (both products are cut off, so that t
  // may be 3 too large: taken off again)
  const uint32_t t = 0x80000000u - mulhi((uint32_t)(d.m >> 21), y0);
  d.y = y0 + mulhi(y0, 2 * t) - 4;
  return d;
}

XF_SLOW double div_plain(double a, double b) { return a / b; }

// a / d.b
XF_FN double div(double a, const Divisor &d) {
  const uint64_t u = bits(a);
  const uint32_t ah = hi32(u);
  if (!(plain_exponent(ah) && plain_exponent(d.h))) {
    // a zero over a plain divisor is the zero of the quotient's sign
    if ((u << 1) == 0 && plain_exponent(d.h))
      return from_bits((uint64_t)((ah ^ d.h) & 0x80000000u) << 32);
    return div_plain(a, d.b);
  }
  uint64_t A = (u & 0x000fffffffffffffull) | 0x0010000000000000ull;
  // A / m in [1, 2)
  const uint32_t less = A < d.m ? 1u : 0u;
  A <<= less;
  // first digit: at most 9 below 2^30 A / m
  const uint32_t d1 = mulhi((uint32_t)(A >> 22), d.y);
  const uint64_t r1 = (A << 30) - mul_digit(d1, d.m);  // < 9 m
  // second digit: less than 1/5 below 2^22 r1 / m (5.3 of its 2^5 cut-off units)
  const uint32_t d2 = mulhi((uint32_t)(r1 >> 25), d.y) >> 5;
  const uint64_t r2 = (r1 << 22) - mul_digit(d2, d.m);  // < 6/5 m
  // q <= A / m 2^52 < q + 6/5, and a quotient is no midpoint: up iff the
  // remainder is over half (a digit one too low has a remainder of m or more)
  const uint64_t q = ((uint64_t)d1 << 22) + d2 + (2 * r2 > d.m ? 1u : 0u);
  // exponent ea - eb - less (+ the bias, one less for q's leading bit)
  const uint32_t e = (ah & 0x7ff00000u) - (d.h & 0x7ff00000u) + (1022u << 20) - (less << 20);
  return from_bits(q + ((uint64_t)(e | ((ah ^ d.h) & 0x80000000u)) << 32));
}
XF_FN double div(double a, double b) { return div(a, divisor(b)); }

XF_SLOW double sqrt_plain(double x) {
#ifdef __CUDA_ARCH__
  return ::sqrt(x);
#else
  return std::sqrt(x);
#endif
}

XF_FN double sqrt_rn(double x) {
  const uint64_t u = bits(x);
  const uint32_t h = hi32(u);
  if (!(h - kLo < kSpan)) {  // a sign bit fails too
    if ((u << 1) == 0) return x;
    return sqrt_plain(x);
  }
  // X in [2^52, 2^54) with an even exponent: sqrt(X 2^52) in [2^52, 2^53)
  const uint32_t odd = 1u - ((h >> 20) & 1u);  // the bias is odd
  const uint64_t X = ((u & 0x000fffffffffffffull) | 0x0010000000000000ull) << odd;
  // y0 = 2^32 / sqrt(X / 2^52), from below (see divisor)
  const float f = float_bits(((uint32_t)(X >> (29 + odd)) & 0x7fffffu) | (0x3f800000u + (odd << 23)));
  float y = seed_rsqrt(f);
  y = at_least_half(y - y * 7.2e-7f);
  const uint32_t y0 = (bits_float(y) << 8) | 0x80000000u;
  // Newton: y1 = y0 (1 + t / 2^31), t / 2^30 = 1 - x y0^2 at most (the three
  // cut-offs in it are worth 3)
  const uint32_t Xh = (uint32_t)(X >> 22);  // 2^30 x
  const uint32_t t3 = 0x40000000u - mulhi(Xh, mulhi(y0, y0));
  const uint32_t t = t3 > 3u ? t3 - 3u : 0u;
  const uint32_t y1 = y0 + mulhi(y0, 2 * t);
  // first digit: at most 6 below 2^30 sqrt(x)
  const uint32_t s1 = mulhi(Xh, y1);
  const uint64_t r1 = (X << 8) - (uint64_t)s1 * s1;  // 2^60 x - s1^2
  // second digit, 2^22 r1 / (2 s1) less its square over 2^23 s1: that is below
  // 2^-28.9 of it, and 8 of y1 are more; in all at most 0.4 too low
  const uint32_t d2 = mulhi((uint32_t)(r1 >> 6), y1 - 8) >> 3;
  const uint64_t s = ((uint64_t)s1 << 22) + d2;
  // 2^104 x - s^2 = 2^44 r1 - 2^23 s1 d2 - d2^2 (mod 2^64)
  const uint64_t r2 = (r1 << 44) - (((uint64_t)s1 * d2) << 23) - (uint64_t)d2 * d2;
  const uint64_t q = s + (r2 > s ? 1u : 0u);
  const uint32_t e = ((((h >> 20) - 1023u - odd) << 19) & 0xfff00000u) + (1022u << 20);
  return from_bits(q + ((uint64_t)e << 32));
}

XF_SLOW double half_plain(double x) { return x * 0.5; }

// x / 2
XF_FN double half(double x) {
  const uint64_t u = bits(x);
  if (plain_exponent(hi32(u))) return from_bits(u - 0x0010000000000000ull);
  if ((u << 1) == 0) return x;
  return half_plain(x);
}

// 0 + x: x, but 0 for -0
XF_FN double plus_zero(double x) {
  return from_bits((bits(x) << 1) == 0 ? 0ull : bits(x));
}

// 0 < x
XF_FN bool positive(double x) { return bits(x) - 1 < 0x7ff0000000000000ull; }

XF_SLOW bool less_plain(double a, double b) { return a < b; }

// a < b; by the bits where both are +0 .. inf (their patterns order like the
// values)
XF_FN bool less(double a, double b) {
  const uint64_t u = bits(a), v = bits(b);
  if (u <= 0x7ff0000000000000ull && v <= 0x7ff0000000000000ull) return u < v;
  return less_plain(a, b);
}

XF_SLOW bool lesseq_plain(double a, double b) { return a <= b; }

// a <= b, likewise
XF_FN bool lesseq(double a, double b) {
  const uint64_t u = bits(a), v = bits(b);
  if (u <= 0x7ff0000000000000ull && v <= 0x7ff0000000000000ull) return u <= v;
  return lesseq_plain(a, b);
}

XF_SLOW double absmaller_plain(double a, double b) {
  const double x = a < 0 ? -a : a, y = b < 0 ? -b : b;
  return a * b <= 0.0 ? 0.0 : (x < y ? a : b);
}

// a b <= 0 ? 0 : (|a| < |b| ? a : b); by signs and magnitudes where the product
// neither vanishes nor overflows, and where one of them is 0
XF_FN double absmaller(double a, double b) {
  const uint64_t u = bits(a), v = bits(b);
  const uint32_t h = hi32(u), k = hi32(v);
  if (plain_exponent(h) && plain_exponent(k))
    return from_bits((int32_t)(h ^ k) < 0 ? 0ull : ((u << 1) < (v << 1) ? u : v));
  const bool fa = (h & 0x7ff00000u) != 0x7ff00000u, fb = (k & 0x7ff00000u) != 0x7ff00000u;
  if (fa && fb && ((u << 1) == 0 || (v << 1) == 0)) return 0.0;
  return absmaller_plain(a, b);
}

// x + p 0
XF_FN double plus_none(double x, double p) {
  const uint32_t h = hi32(bits(p));
  if ((h & 0x7ff00000u) == 0x7ff00000u) return x + p * 0.0;
  return (int32_t)h < 0 ? x : plus_zero(x);
}

}  // namespace xf
}  // namespace om
