// vf_exact.h -- IEEE Float64 operations computed off the FP64 pipe.
//
// GB300 runs Float64 arithmetic at 2 thread instructions per clock and SM
// against 128 issue slots: measured 524 Gop/s for DADD, DMUL and DFMA alike,
// and a DADD with 64 independent integer instructions beside it still runs at
// 502 Gop/s. One Float64 operation costs as much time as about 61 integer
// ones, and the two pipes run side by side, so everything below that is exact
// in integers is cheaper there. Library calls measured 70 (sqrt) and 42 (cbrt)
// Gop/s, i.e. 7.5 and 12 Float64 operations; a comparison, or a conversion
// between Float64 and Float32, costs one.
//
//  half, scale_pow2   products with powers of two, on the exponent field;
//  zero_minus         0 - x;
//  quotient           RN(a/b) by three digits of 21, 20 and 11 bits, each from
//                     a Float32 reciprocal of the divisor, with the remainder
//                     kept exactly in 64 bits (long division in a large radix:
//                     Knuth, TAOCP vol. 2, 4.3.1); about 55 integer and Float32
//                     instructions and no Float64 one, where a correctly
//                     rounded reciprocal and Markstein's residual took 3 of
//                     them per quotient and 5 per divisor;
//  square_root        RN(sqrt(x)) the same way from a Float32 reciprocal root;
//  cube_root_seed     cbrt within a few ulps from a Float32 seed and one
//                     Taylor step in 7 Float64 operations.
//
// All of them return the IEEE result for every operand: operands outside the
// range a method covers (subnormal, infinite, NaN, results near the ends of
// the exponent range) take the Float64 instruction itself.
//
// Plain C++ on the host (with the division and square root of the compiler as
// Float32 seeds), so the integer steps are tested on the CPU.
#pragma once
#include <cstdint>
#include <cstring>

#if defined(__CUDACC__)
#define VF_XFN __device__ __forceinline__
#else
#include <cmath>
#define VF_XFN static inline
#endif

namespace vf {
namespace exact {

using u32 = uint32_t;
using u64 = uint64_t;

#if defined(__CUDACC__)
VF_XFN u64 bits(double x) { return (u64)__double_as_longlong(x); }
VF_XFN double from_bits(u64 b) { return __longlong_as_double((long long)b); }
VF_XFN u32 fbits(float x) { return __float_as_uint(x); }
VF_XFN float ffrom(u32 b) { return __uint_as_float(b); }
VF_XFN float ffma(float a, float b, float c) { return __fmaf_rn(a, b, c); }
VF_XFN float fmulr(float a, float b) { return __fmul_rn(a, b); }
VF_XFN float frcp(float x) {  // at most 1 ulp off
  float y;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
VF_XFN float frsqrt(float x) {  // relative error at most 2^-22.9
  float y;
  asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
VF_XFN float fmcbrt(float x) {  // x^(-1/3), x in [1, 8); relative error below 2^-19
  float l, y;
  asm("lg2.approx.ftz.f32 %0, %1;" : "=f"(l) : "f"(x));
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(l * (-1.0f / 3.0f)));
  return y;
}
VF_XFN double dfma(double a, double b, double c) { return __fma_rn(a, b, c); }
VF_XFN double dmul(double a, double b) { return __dmul_rn(a, b); }
VF_XFN double ddiv(double a, double b) { return __ddiv_rn(a, b); }
VF_XFN double dsqrt(double a) { return __dsqrt_rn(a); }
#else
#ifndef VF_SEED_ULPS  // host tests move the Float32 seeds by this many ulps
#define VF_SEED_ULPS 0
#endif
VF_XFN u64 bits(double x) { u64 b; std::memcpy(&b, &x, 8); return b; }
VF_XFN double from_bits(u64 b) { double x; std::memcpy(&x, &b, 8); return x; }
VF_XFN u32 fbits(float x) { u32 b; std::memcpy(&b, &x, 4); return b; }
VF_XFN float ffrom(u32 b) { float x; std::memcpy(&x, &b, 4); return x; }
VF_XFN float ffma(float a, float b, float c) { return std::fma(a, b, c); }
VF_XFN float fmulr(float a, float b) { return a * b; }
VF_XFN float frcp(float x) { return ffrom(fbits(1.0f / x) + (u32)(VF_SEED_ULPS)); }
VF_XFN float frsqrt(float x) { return ffrom(fbits((float)(1.0 / std::sqrt((double)x))) + (u32)(VF_SEED_ULPS)); }
#ifndef VF_CBRT_SEED_ERROR  // relative
#define VF_CBRT_SEED_ERROR 0
#endif
VF_XFN float fmcbrt(float x) {
  return ffrom(fbits((float)((1.0 + VF_CBRT_SEED_ERROR) / std::cbrt((double)x))) + (u32)(8 * VF_SEED_ULPS));
}
VF_XFN double dfma(double a, double b, double c) { return std::fma(a, b, c); }
VF_XFN double dmul(double a, double b) { return a * b; }
VF_XFN double ddiv(double a, double b) { return a / b; }
VF_XFN double dsqrt(double a) { return std::sqrt(a); }
#endif

// The FP64 product for a path that is hardly ever taken. The compiler turns a
// short branch into predicated instructions, and a predicated-off FP64
// instruction still takes its turn on the pipe; a loop whose trip count it does
// not know stays a branch.
#if defined(__CUDACC__)
static __constant__ int k_one = 1;
#endif
VF_XFN double off_path_mul(double a, double b) {
#if defined(__CUDACC__)
  double r = a;
#pragma unroll 1
  for (int i = 0; i < k_one; ++i) asm volatile("mul.rn.f64 %0, %1, %2;" : "=d"(r) : "d"(a), "d"(b));
  return r;
#else
  return a * b;
#endif
}

VF_XFN u32 hi32(u64 b) { return (u32)(b >> 32); }

// x is +0 or -0. From the two halves of x: a test of the whole word's bits is
// turned into a Float64 comparison by the compiler (20% of the tile kernels'
// FP64 instructions at one time).
VF_XFN bool zero(double x) {
#if defined(__CUDACC__)
  return ((u32)__double2hiint(x) << 1 | (u32)__double2loint(x)) == 0u;
#else
  return (bits(x) << 1) == 0;
#endif
}

// 0.5 * x. Below twice the smallest normal number the bits are a multiple of
// the spacing, and halving them rounds half to even.
VF_XFN double half(double x) {
  const u64 b = bits(x);
  const u32 h = hi32(b) & 0x7ff00000u;
  if (h < 0x00200000u && !zero(x)) {
    const u64 m = b & 0x7fffffffffffffffull, k = m >> 1;
    return from_bits((b & 0x8000000000000000ull) | (k + (m & k & 1)));
  }
  const u32 d = (h - 0x00200000u) < 0x7fd00000u ? 0x00100000u : 0u;  // zero, infinity, NaN stay
  return from_bits(b - ((u64)d << 32));
}

// x * s for s = 2^k: k added to the exponent field where operand and result
// are normal numbers (or zero), else the product.
VF_XFN double scale_pow2(double x, int k, double s) {
  const u64 b = bits(x);
  const int e = (int)((hi32(b) >> 20) & 0x7ff);
  if (zero(x)) return x;
  if (e < 1 || e > 2046 || e + k < 1 || e + k > 2046) return off_path_mul(x, s);
  return from_bits(b + ((u64)((u32)k << 20) << 32));
}

// 0 - x: the sign changed, and +0 for either zero (0 - +0 and 0 - -0 round to +0).
VF_XFN double zero_minus(double x) {
  return from_bits(zero(x) ? 0ull : bits(x) ^ 0x8000000000000000ull);
}

// Divisor of several quotients.
struct Divisor {
  double b;
  u64 D;     // significand, 2^52 <= D < 2^53
  float y;   // about 2^52 / D, in (1/2, 1]
  int e;     // exponent field; outside 1..2046: the IEEE division
};

VF_XFN Divisor divisor(double b) {
  const u64 v = bits(b);
  Divisor d;
  d.b = b;
  d.e = (int)((hi32(v) >> 20) & 0x7ff);
  d.D = (v & 0xfffffffffffffull) | (1ull << 52);
  d.y = frcp(ffrom((u32)(v >> 29 & 0x7fffffu) | 0x3f800000u));
  return d;
}

// RN(a / d.b). With A and D the significands (A doubled when A < D, so the
// quotient q = A/D lies in [1, 2)), every estimate below is a product of
// Float32 numbers added to 2^23, whose low bits are then the rounded integer:
//   Q1 = estimate of q 2^21 less 2: the Float32 operands are off by 2^-23 each
//        and y by another 2^-23, so 0.5 <= q 2^21 - Q1 <= 3.5;
//   Q2 = estimate of (remainder 1) 2^20 / D less 2, off by 0.6 .. 4.4;
//   Q3 = estimate of (remainder 2) 2^11 / D, off by at most 0.51.
// The remainders are exact modulo 2^64 and lie in [0, 5 D); the last one
// decides whether Q3 is the nearest integer or its neighbour is. No quotient
// of two 53-bit significands lies halfway between two 53-bit numbers.
VF_XFN double quotient(const Divisor& d, double a) {
  const u64 v = bits(a);
  const int ea = (int)((hi32(v) >> 20) & 0x7ff);
  u64 A = (v & 0xfffffffffffffull) | (1ull << 52);
  const bool up = A < d.D;
  const int e = ea - d.e + (up ? 1022 : 1023);
  const u32 sign = (hi32(v) ^ hi32(bits(d.b))) & 0x80000000u;
  if (ea < 1 || ea > 2046 || d.e < 1 || d.e > 2046 || e < 1 || e > 2046) {
    if (zero(a) && d.e >= 1 && d.e <= 2046) return from_bits((u64)sign << 32);
    return ddiv(a, d.b);
  }
  const float af = ffrom((u32)(v >> 29 & 0x7fffffu) | (up ? 0x40000000u : 0x3f800000u));
  if (up) A <<= 1;
  const u32 q1 = fbits(ffma(af, fmulr(d.y, 2097152.0f), 8388608.0f)) - (0x4b000000u + 2u);
  const u64 r1 = (A << 21) - (u64)q1 * d.D;
  const u32 q2 = fbits(ffma((float)hi32(r1), d.y, 8388608.0f)) - (0x4b000000u + 2u);
  const u64 r2 = (r1 << 20) - (u64)q2 * d.D;
  u32 q3 = fbits(ffma((float)hi32(r2), fmulr(d.y, 0x1p-9f), 8388608.0f)) - 0x4b000000u;
  const long long r3 = (long long)((r2 << 11) - (u64)q3 * d.D);
  const long long t = r3 + r3, D = (long long)d.D;
  q3 += (t > D ? 1u : 0u) - (t < -D ? 1u : 0u);
  const u64 q = ((u64)q1 << 31) + ((u64)q2 << 11) + q3;
  return from_bits(q - (1ull << 52) + ((u64)(((u32)e << 20) | sign) << 32));
}

// RN(sqrt(x)): x = X 2^(2k) with 2^52 <= X < 2^54, s = sqrt(X / 2^52) in [1, 2).
//   S1 = estimate of s 2^21 less 2: off by 0.7 .. 3.3 (y is off by 2^-22.4);
//   S2 = S1 2^20 + (estimate of its error less 2): off by 0.8 .. 6.9, the
//        neglected square of the error included;
//   S  = S2 2^11 + estimate of its error: off by at most 0.51.
// The remainders X 2^2j - S^2 are exact; S is the nearest integer when the
// last lies in (-S, S]. No root lies halfway between two 53-bit numbers.
VF_XFN double square_root(double x) {
  const u64 v = bits(x);
  const int ex = (int)(hi32(v) >> 20);  // with the sign bit: negative numbers are out of range
  if (ex < 1 || ex > 2046) return zero(x) ? x : dsqrt(x);
  const bool odd = (ex & 1) == 0;  // unbiased exponent odd
  u64 X = (v & 0xfffffffffffffull) | (1ull << 52);
  const float xf = ffrom((u32)(v >> 29 & 0x7fffffu) | (odd ? 0x40000000u : 0x3f800000u));
  if (odd) X <<= 1;
  const float y = frsqrt(xf);
  const u32 s1 = fbits(ffma(xf, fmulr(y, 2097152.0f), 8388608.0f)) - (0x4b000000u + 2u);
  const u64 r1 = X - ((u64)s1 * s1 << 10);
  const u32 q2 = fbits(ffma((float)(u32)(r1 >> 12), y, 8388608.0f)) - (0x4b000000u + 2u);
  const u64 r2 = (r1 << 30) - (u64)q2 * (((u64)s1 << 21) + q2);
  const u64 s2 = ((u64)s1 << 20) + q2;
  const u32 q3 = fbits(ffma((float)(u32)(r2 >> 23), fmulr(y, 0x1p-8f), 8388608.0f)) - 0x4b000000u;
  const long long r3 = (long long)((r2 << 22) - (u64)q3 * ((s2 << 12) + q3));
  long long s = (long long)((s2 << 11) + q3);
  s += (r3 > s ? 1 : 0) - (r3 <= -s ? 1 : 0);
  const u32 e = (u32)((ex - 1023) >> 1) + 1023u;
  return from_bits((u64)s - (1ull << 52) + ((u64)(e << 20) << 32));
}

// cbrt(t) for t in [1, 8), within 5.3 units of 2^-53 relative: with w ~ t^(-1/3)
// and e = 1 - t w^3, cbrt(t) = t w^2 (1 - e)^(-2/3). A w off by 2^-19 gives
// |e| < 3.01 2^-19, and the Taylor series after e^2 leaves 40/81 e^3 < 0.85 2^-53;
// the roundings of t w, w^2 and c add 2 units through c and 4/3 through e, the
// last sum another. cr_cbrt finds the nearest double by exact comparisons.
VF_XFN double cube_root_seed(double t) {
  const u64 v = bits(t);
  // Float32 value of t by its bits (a conversion instruction runs on the FP64 pipe)
  const float tf = ffrom((u32)(v >> 29) - (896u << 23));
  const double w = from_bits(((u64)fbits(fmcbrt(tf)) << 29) + ((u64)896u << 52));
  const double tw = dmul(t, w);
  const double e = dfma(-tw, dmul(w, w), 1.0);
  const double c = dmul(tw, w);
  return dfma(c, dmul(dfma(e, 5.0 / 9.0, 2.0 / 3.0), e), c);
}

}  // namespace exact
}  // namespace vf
