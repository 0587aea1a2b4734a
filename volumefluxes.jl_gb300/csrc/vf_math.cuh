// vf_math.cuh -- per-cell and per-face arithmetic of VolumeFluxes.jl's
// practical 2D shallow-water path, restated for the device.
//
// Every expression keeps the reference's operation order, because the Float64
// path must reproduce the reference bit for bit: the Float64 translation unit
// is compiled with -fmad=false, so a*b+c stays two rounded operations as in
// Julia. Float32 instances may contract and use fast reciprocals (their error
// is stated against the Float64 oracle, not claimed bitwise).
//
// GB300 executes Float64 at 1/64 of the Float32 rate, so the Float64 traits
// below move every comparison, min/max and sign test onto the integer pipe by
// comparing IEEE bit patterns, and quotients, square roots and products with
// powers of two by computing them in integers (vf_exact.h); only +, -, * stay
// on the FP64 pipe.
//
// Citations are path:line within the VolumeFluxes.jl project.
#pragma once
#include <cstdint>
#include <type_traits>
#include <cuda_runtime.h>

#include "vf_exact.h"

// Float32 reciprocals and cube roots come from the special-function unit
// (rcp.approx, and cbrt(x) = 2^(log2|x| / 3) with the sign of x; a few ulps);
// Float32 results are stated against the Float64 oracle, not claimed bitwise.
// Measured on the 4096^2 wet/dry step (Float32 is instruction-issue bound):
// 0.919 ms with the special-function unit, 1.069 ms with the correctly
// rounded reciprocal and the libm cube root.
// 1 (vf_f64f.cu): the tolerance-bound Float64 kernels, whose face fluxes use
// fused multiply-adds. 0: every operation rounds as in the reference (the
// bitwise kernels). Quotients, square roots and cube roots are the correctly
// rounded ones of vf_exact.h in both: they cost no FP64 instructions.
#ifndef VF_FP64_FAITHFUL
#define VF_FP64_FAITHFUL 0
#endif

namespace vf {

// ---------------------------------------------------------------------------
// Precision traits.
template <typename T>
struct Arith;

// Float64: exact IEEE semantics. Comparisons are done on bit patterns (valid
// for every non-NaN operand; a valid step never produces NaN because every
// divisor is bounded away from zero).
template <>
struct Arith<double> {
  static constexpr bool exact = !VF_FP64_FAITHFUL;
  static __device__ __forceinline__ long long bits(double x) { return __double_as_longlong(x); }
  // Monotone key: orders all non-NaN doubles, with -0.0 just below +0.0.
  static __device__ __forceinline__ long long key(double x) {
    const long long b = bits(x);
    return b ^ ((b >> 63) & 0x7fffffffffffffffll);
  }
  static __device__ __forceinline__ bool both_zero(double x, double y) {
    return ((unsigned long long)(bits(x) | bits(y)) << 1) == 0ull;
  }
  static __device__ __forceinline__ bool lt(double x, double y) { return key(x) < key(y) && !both_zero(x, y); }
  static __device__ __forceinline__ bool gt(double x, double y) { return key(x) > key(y) && !both_zero(x, y); }
  static __device__ __forceinline__ bool gt0(double x) { return __double2hiint(x) >= 0 && !exact::zero(x); }
  static __device__ __forceinline__ bool lt0(double x) { return __double2hiint(x) < 0 && !exact::zero(x); }
  // |x| < k and |x| >= k for k >= 0.
  static __device__ __forceinline__ bool abs_lt(double x, double k) {
    return (unsigned long long)(bits(x) & 0x7fffffffffffffffll) < (unsigned long long)bits(k);
  }
  static __device__ __forceinline__ bool is_zero(double x) { return exact::zero(x); }
  // Julia's max/min: -0.0 < +0.0.
  static __device__ __forceinline__ double max(double x, double y) { return key(x) > key(y) ? x : y; }
  static __device__ __forceinline__ double min(double x, double y) { return key(x) < key(y) ? x : y; }
  // Correctly rounded quotients and square roots in integers (vf_exact.h):
  // the IEEE bits without an FP64 instruction, about 55 integer and Float32
  // instructions each.
  using Recip = exact::Divisor;
  static __device__ __forceinline__ Recip recip(double b) { return exact::divisor(b); }
  static __device__ __forceinline__ double div_by(const Recip& R, double a) { return exact::quotient(R, a); }
  static __device__ __forceinline__ double div(double a, double b) { return div_by(recip(b), a); }
  static __device__ __forceinline__ double rcp(double b) { return div(1.0, b); }
  static __device__ __forceinline__ double inv(const Recip& R) { return div_by(R, 1.0); }
  static __device__ __forceinline__ double sqrt_(double x) { return exact::square_root(x); }
};

template <>
struct Arith<float> {
  static constexpr bool exact = false;
  static __device__ __forceinline__ bool lt(float x, float y) { return x < y; }
  static __device__ __forceinline__ bool gt(float x, float y) { return x > y; }
  static __device__ __forceinline__ bool gt0(float x) { return x > 0.f; }
  static __device__ __forceinline__ bool lt0(float x) { return x < 0.f; }
  static __device__ __forceinline__ bool abs_lt(float x, float k) { return fabsf(x) < k; }
  static __device__ __forceinline__ bool is_zero(float x) { return x == 0.f; }
  static __device__ __forceinline__ float max(float x, float y) { return fmaxf(x, y); }
  static __device__ __forceinline__ float min(float x, float y) { return fminf(x, y); }
  static __device__ __forceinline__ float div(float a, float b) { return __fdividef(a, b); }
  static __device__ __forceinline__ float rcp(float b) { return __fdividef(1.0f, b); }
  static __device__ __forceinline__ float sqrt_(float x) { return sqrtf(x); }
  // Quotients over one divisor: one reciprocal, then products.
  struct Recip {
    float r;
  };
  static __device__ __forceinline__ Recip recip(float b) { return Recip{rcp(b)}; }
  static __device__ __forceinline__ float div_by(const Recip& R, float a) { return a * R.r; }
  static __device__ __forceinline__ float inv(const Recip& R) { return R.r; }
};

// ---------------------------------------------------------------------------
// Correctly rounded cube root (Float64). A seed within a few ulps (eight at most)
// is corrected with an exact integer comparison against the rounding midpoints, so
// the result is the nearest double regardless of the seed's last-bit error; the
// CPU oracle computes the same unique value.
__device__ __forceinline__ void cube_u55(uint64_t k, uint64_t& w0, uint64_t& w1, uint64_t& w2) {
  const uint64_t lo = k * k, hi = __umul64hi(k, k);       // k^2 < 2^110
  const uint64_t p0lo = k * lo, p0hi = __umul64hi(k, lo);  // k*lo < 2^119
  const uint64_t p1lo = k * hi, p1hi = __umul64hi(k, hi);  // k*hi < 2^101
  w0 = p0lo;
  w1 = p0hi + p1lo;
  w2 = p1hi + (w1 < p1lo ? 1ull : 0ull);
}
__device__ __forceinline__ int cmp192(uint64_t a0, uint64_t a1, uint64_t a2, uint64_t b0, uint64_t b1, uint64_t b2) {
  if (a2 != b2) return a2 < b2 ? -1 : 1;
  if (a1 != b1) return a1 < b1 ? -1 : 1;
  if (a0 != b0) return a0 < b0 ? -1 : 1;
  return 0;
}

// Out of line: the friction law calls it from two places per cell and step
// (inlined it measured 31.06 vs 31.00 ms per 4096^2 wet/dry step).
static __device__ __noinline__ double cr_cbrt(double x) {
  const uint64_t sign = exact::bits(x) & 0x8000000000000000ull;
  uint64_t bits = exact::bits(x) ^ sign;
  if (bits == 0 || bits >= 0x7ff0000000000000ull) return x;
  int extra = 0;
  if ((bits >> 52) == 0) {
    bits = exact::bits(exact::from_bits(bits) * 18014398509481984.0);  // 2^54, exact
    extra = 18;
  }
  const int e = (int)(bits >> 52) - 1023;
  const uint64_t frac = bits & ((1ull << 52) - 1);
  const uint64_t M = frac | (1ull << 52);
  const int q = e >= 0 ? e / 3 : -((-e + 2) / 3);
  const int r = e - 3 * q;  // 0, 1, 2
  const double t = __longlong_as_double((long long)(((uint64_t)(1023 + r) << 52) | frac));  // in [1, 8)
  const uint64_t y0 = exact::bits(exact::cube_root_seed(t));
  uint64_t Y;
  if (y0 >= 0x4000000000000000ull) {         // 2
    Y = 1ull << 53;
  } else if (y0 < 0x3ff0000000000000ull) {   // 1
    Y = 1ull << 52;
  } else {
    Y = (y0 & ((1ull << 52) - 1)) | (1ull << 52);
  }
  // t * 2^159 = M * 2^(r + 107): limbs (0, M << (43 + r), M >> (21 - r)).
  const uint64_t T1 = M << (43 + r), T2 = M >> (21 - r);
  for (int it = 0; it < 8; ++it) {
    uint64_t c0, c1, c2;
    cube_u55(2 * Y + 1, c0, c1, c2);
    if (cmp192(c0, c1, c2, 0, T1, T2) < 0) { ++Y; continue; }
    if (Y > (1ull << 52)) {
      cube_u55(2 * Y - 1, c0, c1, c2);
      if (cmp192(c0, c1, c2, 0, T1, T2) > 0) { --Y; continue; }
    }
    break;
  }
  // y = Y * 2^(q - 52 - extra), Y in [2^52, 2^53].
  int ex = q - extra;
  uint64_t mant = Y;
  if (mant == (1ull << 53)) { mant >>= 1; ex += 1; }
  return exact::from_bits(((uint64_t)(ex + 1023) << 52) | (mant & ((1ull << 52) - 1)) | sign);
}

template <typename T> __device__ __forceinline__ T vcbrt(T x);
template <> __device__ __forceinline__ double vcbrt<double>(double x) { return cr_cbrt(x); }
template <> __device__ __forceinline__ float vcbrt<float>(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(__log2f(fabsf(x)) * (1.0f / 3.0f)));
  return copysignf(y, x);
}

// Back-compat names used by the tile kernels.
template <typename T> __device__ __forceinline__ T jmax(T x, T y) { return Arith<T>::max(x, y); }
template <typename T> __device__ __forceinline__ T jmin(T x, T y) { return Arith<T>::min(x, y); }
template <typename T> __device__ __forceinline__ T vdiv(T a, T b) { return Arith<T>::div(a, b); }

// x/2 and x/4: for Float64 on the exponent field (the same bits).
template <typename T> __device__ __forceinline__ T halve(T x) {
  if constexpr (std::is_same<T, double>::value) return exact::half(x);
  else return (T)0.5 * x;
}
template <typename T> __device__ __forceinline__ T quarter(T x) {
  // halving twice rounds as a quarter does: x/2 is inexact only where its last
  // place is the smallest there is, and rounds to even there
  if constexpr (std::is_same<T, double>::value) return exact::half(exact::half(x));
  else return (T)0.25 * x;
}
// a*b + c and a*b - c of the face fluxes: one rounding in the tolerance-bound
// Float64 kernels, two (as the reference's) in the bitwise ones; other types
// as their unit's contraction setting has it.
template <typename T> __device__ __forceinline__ T madd(T a, T b, T c) {
  if constexpr (std::is_same<T, double>::value && VF_FP64_FAITHFUL) return __fma_rn(a, b, c);
  else return a * b + c;
}
template <typename T> __device__ __forceinline__ T msub(T a, T b, T c) {
  if constexpr (std::is_same<T, double>::value && VF_FP64_FAITHFUL) return __fma_rn(a, b, -c);
  else return a * b - c;
}
// The larger of two speeds >= 0, ignoring a NaN in v.
template <typename T> __device__ __forceinline__ T speed_max(T m, T v) {
  if constexpr (std::is_same<T, double>::value) {
    const long long b = __double_as_longlong(v);
    return b > __double_as_longlong(m) && b <= 0x7ff0000000000000ll ? v : m;
  } else {
    return fmax(m, v);
  }
}

// ---------------------------------------------------------------------------
// Physical constants of one simulation in the state's real type.
template <typename T>
struct Phys {
  T g, neg_g, rho, c2;        // c2 = (0.5*rho)*g, as Julia folds 0.5*ρ*g*h^2
  T cutoff, kappa, theta;
  T inv_dx, inv_dy;           // 1/Δx, 1/Δy (src/numericalflux/numericalflux.jl:27)
  T dx, dy;                   // Δx, Δy (src/sourceterms/source_term_bottom.jl:38)
  int dx_pow2, dy_pow2;       // Δ is a power of two: x/Δ == x*(1/Δ) exactly
  int dx_exp, dy_exp;         // then 1/Δ == 2^exp
  int unit_rho;               // rho == 1: rho*h == h exactly
  T Cz;
  T near_dry;                 // Float32: |h| below this takes the Float64 velocity division (0: never)
  int friction;               // VF_FRICTION_*
  int n_bottom;               // SourceTermBottom entries
  int n_point;                // rain/infiltration entries, applied in order
  int rec_none;               // NoReconstruction instead of LinearReconstruction
  int any_dynamic;            // some point source is not a constant
  int point_kind[8];          // PointKind
  T point_add[8];             // kConstant: +rate/3600 for rain, -rate for infiltration
  T point_sum;                // Float32: the constant point sources' sum (summed in Float64)
  T bottom_g;                 // Float32: n_bottom * (-g), the bottom sources' factor at once
  T half_over_kappa;          // Float32: 0.5 / kappa
  const T* point_field[8];    // kHorton: factor, kField: rain rate [m/s]; total grid, state layout
  int n_fields;               // Float32: sources with a field, in order
  const T* field[8];          // Float32: their fields
  const double* tab_t[8];     // kTable: breakpoints of TimeDependentRain
  const double* tab_r[8];     // kTable: rates/3600 per breakpoint
  int tab_n[8];
  double horton[8][3];        // kHorton: fc, f0, k
};

enum PointKind { kConstant = 0, kTable = 1, kHorton = 2, kField = 3 };

// Deterministic exp for HortonInfiltration: Cody-Waite reduction by ln 2 (split
// in two doubles), Taylor polynomial of degree 14 in Horner form with fused
// multiply-adds, exact scaling by 2^k. The oracle computes the same bits.
__device__ __forceinline__ double det_exp(double x) {
  if (x != x) return x;
  if (x > 709.782712893384) return __longlong_as_double(0x7ff0000000000000ll);
  if (x < -745.1332191019412) return 0.0;
  const double inv_ln2 = 0x1.71547652b82fep+0;
  const double ln2_hi = 0x1.62e42fefa39efp-1, ln2_lo = 0x1.abc9e3b39803fp-56;
  double kd = x * inv_ln2;
  kd = (kd + 6755399441055744.0) - 6755399441055744.0;  // round to nearest integer
  double r = fma(-kd, ln2_hi, x);
  r = fma(-kd, ln2_lo, r);
  const double c[15] = {0x1.0000000000000p+0, 0x1.0000000000000p+0, 0x1.0000000000000p-1,
                        0x1.5555555555555p-3, 0x1.5555555555555p-5, 0x1.1111111111111p-7,
                        0x1.6c16c16c16c17p-10, 0x1.a01a01a01a01ap-13, 0x1.a01a01a01a01ap-16,
                        0x1.71de3a556c734p-19, 0x1.27e4fb7789f5cp-22, 0x1.ae64567f544e4p-26,
                        0x1.1eed8eff8d898p-29, 0x1.6124613a86d09p-33, 0x1.93974a8c07c9dp-37};
  double q = c[14];
#pragma unroll
  for (int n = 13; n >= 0; --n) q = fma(q, r, c[n]);
  int k = (int)kd;
  if (k > 1023) { q = q * 2.0; k -= 1; }
  if (k < -1022) return (q * __longlong_as_double((long long)(k + 54 + 1023) << 52)) * 0x1p-54;
  return q * __longlong_as_double((long long)(k + 1023) << 52);
}

// Per-step scalars of the time-dependent point sources at the step's start
// time t (the same t for both RK2 stages, src/system.jl:71-73):
// TimeDependentRain's tabulated rate (src/sourceterms/source_term_rain.jl:45-54)
// and Horton's fc + (f0 - fc)*exp(-k*t) (src/sourceterms/source_term_infiltration.jl:68-70).
// Float64: one scalar per source, added in list order. Float32: the sum of all
// that are the same in every cell (summed in Float64) in out[0], then one factor
// per source with a field, so a cell adds one scalar and its fields.
constexpr int kScalars = 9;
template <typename T>
__device__ __forceinline__ void point_scalars(const Phys<T>& p, double t, T* out) {
  double sum = 0.0;
  int field = 1;
#pragma unroll 1
  for (int n = 0; n < p.n_point; ++n) {
    double rate = 0.0;
    if (sizeof(T) == 8) out[n] = (T)0;
    if (p.point_kind[n] == kConstant) {
      rate = (double)p.point_add[n];
    } else if (p.point_kind[n] == kTable) {
      int idx = 0;
      while (idx + 1 < p.tab_n[n] && !(t < p.tab_t[n][idx + 1])) ++idx;
      rate = p.tab_r[n][idx];
      if (sizeof(T) == 8) out[n] = (T)rate;
    } else if (p.point_kind[n] == kHorton) {
      const T fc = (T)p.horton[n][0], f0 = (T)p.horton[n][1], k = (T)p.horton[n][2];
      const T decay = (T)det_exp((double)(-k * (T)t));
      const T f = fc + (f0 - fc) * decay;
      if (sizeof(T) == 8) out[n] = f;
      else out[field++] = -f;
    } else if (sizeof(T) == 4) {
      out[field++] = (T)1;
    }
    sum += rate;
  }
  if (sizeof(T) == 4) out[0] = (T)sum;
}

// ΔB/Δ of the bottom source; exact reciprocal multiply when Δ is a power of two.
// Float32 always multiplies by 1/Δ (one rounding more where Δ is not a power
// of two; a 1.5% faster Float32 step, the same bits on power-of-two cells).
template <typename T>
__device__ __forceinline__ T slope_over(T dB, T delta, T inv_delta, int pow2) {
  if constexpr (sizeof(T) == 4) return dB * inv_delta;
  return pow2 ? dB * inv_delta : Arith<T>::div(dB, delta);
}

// v[j] * (1/Δ) along DIR in Float64: for a power-of-two Δ on the exponent field
// (nothing where Δ is 1), the same bits as the products.
template <int DIR, int N>
__device__ __forceinline__ void over_delta(const Phys<double>& p, double (&v)[N]) {
  const double inv = DIR == 0 ? p.inv_dx : p.inv_dy;
  if (DIR == 0 ? p.dx_pow2 : p.dy_pow2) {
    const int k = DIR == 0 ? p.dx_exp : p.dy_exp;
    if (k != 0) {
#pragma unroll
      for (int j = 0; j < N; ++j) v[j] = exact::scale_pow2(v[j], k, inv);
    }
    return;
  }
#pragma unroll
  for (int j = 0; j < N; ++j) v[j] = exact::off_path_mul(inv, v[j]);
}
// The bottom source's slope ΔB/Δ along DIR in the tile kernels.
template <typename T, int DIR>
__device__ __forceinline__ T bottom_slope(const Phys<T>& p, T dB) {
  if constexpr (std::is_same<T, double>::value) {
    if (DIR == 0 ? p.dx_pow2 : p.dy_pow2) {
      double v[1] = {dB};
      over_delta<DIR>(p, v);
      return v[0];
    }
    return Arith<T>::div(dB, DIR == 0 ? p.dx : p.dy);
  } else {
    return slope_over<T>(dB, DIR == 0 ? p.dx : p.dy, DIR == 0 ? p.inv_dx : p.inv_dy, DIR == 0 ? p.dx_pow2 : p.dy_pow2);
  }
}

// Rain and infiltration in list order (src/system.jl:71-73), unrolled so the
// parameter block is never indexed dynamically. `scal` holds point_scalars();
// `cell` is the cell's offset in the state layout (for per-cell arrays).
// Float32 (the marching kernels' constant sources) adds their sum at once:
// one add instead of eight guarded ones, 2-4% of the Float32 stage pass; the
// sum rounds once to Float32 where the list order would round after each
// source (Float32 results are held to a stated error, not to the bits).
template <typename T>
__device__ __forceinline__ T add_point_sources(const Phys<T>& p, T acc0) {
  if constexpr (sizeof(T) == 4) {
    return acc0 + p.point_sum;
  } else {
#pragma unroll 1
    for (int n = 0; n < p.n_point; ++n) acc0 = acc0 + p.point_add[n];
    return acc0;
  }
}
template <typename T>
__device__ __forceinline__ T add_point_sources(const Phys<T>& p, T acc0, const T* scal, long long cell) {
  if constexpr (sizeof(T) == 4) {
    // scal[0]: every source that is the same in all cells; then the fields' factors
    acc0 = acc0 + scal[0];
#pragma unroll 1
    for (int n = 0; n < p.n_fields; ++n) acc0 = acc0 + p.field[n][cell] * scal[1 + n];
    return acc0;
  }
#pragma unroll
  for (int n = 0; n < 8; ++n) {
    if (n >= p.n_point) continue;
    switch (p.point_kind[n]) {
      case kConstant: acc0 = acc0 + p.point_add[n]; break;
      case kTable: acc0 = acc0 + scal[n]; break;
      case kHorton: acc0 = acc0 - p.point_field[n][cell] * scal[n]; break;
      default: acc0 = acc0 + p.point_field[n][cell]; break;
    }
  }
  return acc0;
}

// desingularize, src/equations/equation.jl:40-62 (Eq. 26 of Brodtkorb & Holm 2021).
// For |h| >= kappa the expression equals h exactly: min(...) <= kappa <= |h|.
template <typename T>
__device__ __forceinline__ T desing(T h, T kappa) {
  using A = Arith<T>;
  if (!A::abs_lt(h, kappa)) return h;
  const T m = A::min(A::div(h * h, (T)2 * kappa) + kappa / (T)2, kappa);
  return copysign((T)1, h) * A::max(fabs(h), m);
}

// The Float64 quotient a/b of two Float32 values, rounded to Float32, without
// Float64 instructions. Rounding an IEEE quotient to 53 bits and then to 24
// gives the same bits as rounding it to 24 bits once, because 53 >= 2*24
// (Figueroa, "When is double rounding innocuous?", SIGNUM Newsl. 30(3), 1995),
// so RN32(RN64(a/b)) is the correctly rounded Float32 quotient, which
// __fdiv_rn computes on the Float32 pipes whatever the -prec-div setting. The
// kernels divide near-dry velocities with it: GB300 runs Float64 at 1/64 of
// the Float32 rate, so the Float64 instructions cost a divergent warp several
// hundred cycles per quotient. vf_selftest_near_dry_quotients checks the
// equality against the IEEE Float64 division on the device.
__device__ __forceinline__ float f64_quotient_f32(float a, float b) { return __fdiv_rn(a, b); }

// Desingularised velocities (hu, hv) / h* (src/equations/equation.jl:40-67).
// A Float32 state takes the Float64 quotient (f64_quotient_f32) where
// |h| < p.near_dry, the thin films at wet/dry fronts, and one fast reciprocal
// elsewhere; Float64 divides in its own type.
template <typename T>
__device__ __forceinline__ void velocities(const Phys<T>& p, T h, T hs, T hu, T hv, T& u, T& v) {
  using A = Arith<T>;
  if constexpr (sizeof(T) == 4) {
    if (A::abs_lt(h, p.near_dry)) {
      u = f64_quotient_f32(hu, hs);
      v = f64_quotient_f32(hv, hs);
      return;
    }
  }
  const typename A::Recip R = A::recip(hs);
  u = A::div_by(R, hu);
  v = A::div_by(R, hv);
}

// One side of a face: physical flux (src/equations/swe_2D.jl:43-65) and the
// two outer eigenvalues (src/equations/swe_2D.jl:69-81).
template <typename T, int DIR>
__device__ __forceinline__ void side_flux(const Phys<T>& p, T h, T hu, T hv, T& f0, T& f1, T& f2, T& l1, T& l2) {
  using A = Arith<T>;
  const T hs = desing<T>(h, p.kappa);
  T u, v;
  velocities<T>(p, h, hs, hu, hv, u, v);
  T rh = h;
  if constexpr (std::is_same<T, double>::value) {
    if (!p.unit_rho) rh = exact::off_path_mul(p.rho, h);
  } else {
    rh = p.rho * h;
  }
  const T hh = h * h;
  if (DIR == 0) {
    f0 = rh * u;
    f1 = madd<T>(f0, u, p.c2 * hh);
    f2 = f0 * v;
  } else {
    f0 = rh * v;
    f1 = (rh * u) * v;
    f2 = madd<T>(f0, v, p.c2 * hh);
  }
  const T c = A::sqrt_(p.g * h);
  const T un = DIR == 0 ? u : v;
  l1 = un + c;
  l2 = un - c;
}

// One side of a Float32 face without branches: a dry side takes depth and
// velocities zero, so its flux and eigenvalues come out as zeros. wet: the
// side's depth exceeds the cutoff.
template <int DIR>
__device__ __forceinline__ void side_flux_f32(const Phys<float>& p, bool wet, float h, float u, float v,
                                              float& f0, float& f1, float& f2, float& l1, float& l2) {
  const float hz = wet ? h : 0.f;
  const float rh = p.rho * hz;
  const float hh = hz * hz;
  const float un = DIR == 0 ? u : v;
  f0 = rh * un;
  if (DIR == 0) {
    f1 = f0 * u + p.c2 * hh;
    f2 = f0 * v;
  } else {
    f1 = (rh * u) * v;
    f2 = f0 * v + p.c2 * hh;
  }
  const float c = sqrtf(p.g * hz);
  l1 = un + c;
  l2 = un - c;
}

// cu_face for Float32. Branches cost the issue-bound marching kernels more than
// the work they skip: their own instructions, the zeros for the path not taken,
// and constants loaded anew on each side (the uniform registers are not
// available to divergent code).
template <int DIR, bool SPEED>
__device__ __forceinline__ void cu_face_f32(const Phys<float>& p, float mh, float mhu, float mhv, float ph, float phu,
                                            float phv, float& F0, float& F1, float& F2, float& speed) {
  using A = Arith<float>;
  const bool wm = mh > p.cutoff, wp = ph > p.cutoff;
  // h* = max(h, min(h^2 / (2 kappa) + kappa/2, kappa)) for h > 0 (src/equations/equation.jl:40-62)
  const float hm = fmaxf(mh, fminf(mh * mh * p.half_over_kappa + p.kappa * 0.5f, p.kappa));
  const float hp = fmaxf(ph, fminf(ph * ph * p.half_over_kappa + p.kappa * 0.5f, p.kappa));
  const float rm = A::rcp(hm), rp = A::rcp(hp);
  // selects, not products with zero: a dry side's momentum may be infinite or NaN
  float mu = wm ? mhu * rm : 0.f, mv = wm ? mhv * rm : 0.f, pu = wp ? phu * rp : 0.f, pv = wp ? phv * rp : 0.f;
  const bool nm = wm && mh < p.near_dry, np = wp && ph < p.near_dry;
  if (nm || np) {  // thin films take the Float64 quotient's bits
    if (nm) {
      mu = f64_quotient_f32(mhu, hm);
      mv = f64_quotient_f32(mhv, hm);
    }
    if (np) {
      pu = f64_quotient_f32(phu, hp);
      pv = f64_quotient_f32(phv, hp);
    }
  }
  float fm0, fm1, fm2, em1, em2, fp0, fp1, fp2, ep1, ep2;
  side_flux_f32<DIR>(p, wm, mh, mu, mv, fm0, fm1, fm2, em1, em2);
  side_flux_f32<DIR>(p, wp, ph, pu, pv, fp0, fp1, fp2, ep1, ep2);
  const float aplus = fmaxf(fmaxf(ep1, em1), 0.f);
  const float aminus = fminf(fminf(ep2, em2), 0.f);
  const float d = aplus - aminus;
  const bool waves = !(d < p.kappa);
  const float R = waves || !SPEED ? A::rcp(d) : 0.f;
  const float q = (aplus * aminus) * R;
  const float g0 = (aplus * fm0 - aminus * fp0) * R + q * (ph - mh);
  const float g1 = (aplus * fm1 - aminus * fp1) * R + q * (phu - mhu);
  const float g2 = (aplus * fm2 - aminus * fp2) * R + q * (phv - mhv);
  // No waves, no flux, whatever the values are: zero times a difference that is
  // infinite or NaN would not be zero. The two forms are the faster one of either
  // pass (us per 4096^2 wet/dry launch, flux and stage: assignment 253 and 385,
  // selects 262 and 373; selects around the whole expressions 280 and 389).
  if constexpr (SPEED) {
    F0 = g0, F1 = g1, F2 = g2;
    if (!waves) F0 = F1 = F2 = 0.f;
    speed = waves ? fmaxf(aplus, -aminus) : 0.f;  // waves: one side at least is wet
  } else {
    F0 = waves ? g0 : 0.f;
    F1 = waves ? g1 : 0.f;
    F2 = waves ? g2 : 0.f;
  }
}

// Central-upwind flux across one face, src/numericalflux/swe/centralupwind.jl:48-77.
// minus = right face value of the left cell, plus = left face value of the right cell.
template <typename T, int DIR, bool SPEED>
__device__ __forceinline__ void cu_face(const Phys<T>& p, T mh, T mhu, T mhv, T ph, T phu, T phv, T& F0, T& F1, T& F2,
                                        T& speed) {
  using A = Arith<T>;
  if constexpr (std::is_same<T, float>::value) {
    cu_face_f32<DIR, SPEED>(p, mh, mhu, mhv, ph, phu, phv, F0, F1, F2, speed);
    return;
  }
  T fm0 = 0, fm1 = 0, fm2 = 0, em1 = 0, em2 = 0;
  if (A::gt(mh, p.cutoff)) side_flux<T, DIR>(p, mh, mhu, mhv, fm0, fm1, fm2, em1, em2);
  T fp0 = 0, fp1 = 0, fp2 = 0, ep1 = 0, ep2 = 0;
  if (A::gt(ph, p.cutoff)) side_flux<T, DIR>(p, ph, phu, phv, fp0, fp1, fp2, ep1, ep2);
  const T aplus = A::max(A::max(ep1, em1), (T)0);
  const T aminus = A::min(A::min(ep2, em2), (T)0);
  const T d = aplus - aminus;
  if (A::abs_lt(d, p.kappa)) {
    F0 = F1 = F2 = (T)0;
    if (SPEED) speed = (T)0;
    return;
  }
  const typename A::Recip R = A::recip(d);
  const T q = A::div_by(R, aplus * aminus);
  F0 = madd<T>(q, ph - mh, A::div_by(R, msub<T>(aplus, fm0, aminus * fp0)));
  F1 = madd<T>(q, phu - mhu, A::div_by(R, msub<T>(aplus, fm1, aminus * fp1)));
  F2 = madd<T>(q, phv - mhv, A::div_by(R, msub<T>(aplus, fm2, aminus * fp2)));
  if (SPEED)
    speed = (A::lt(mh, p.cutoff) && A::lt(ph, p.cutoff)) ? (T)0 : A::max(fabs(aplus), fabs(aminus));
}

// minmod and minmod_slope, src/reconstruction/linearreconstruction.jl:28-43.
template <typename T>
__device__ __forceinline__ T minmod(T a, T b, T c) {
  using A = Arith<T>;
  if (A::gt0(a) && A::gt0(b) && A::gt0(c)) return A::min(A::min(a, b), c);
  if (A::lt0(a) && A::lt0(b) && A::lt0(c)) return A::max(A::max(a, b), c);
  return (T)0;
}
// Float32: the same function as max(min(a, b, c), 0) + min(max(a, b, c), 0),
// six min/max and an add instead of six compares and selects (the Float32
// kernels are instruction-issue bound: 1.007 instead of 1.083 ms per 4096^2
// wet/dry step, the same error against Float64). Float64 keeps the
// reference's branches on bit patterns.
template <>
__device__ __forceinline__ float minmod<float>(float a, float b, float c) {
  return fmaxf(fminf(fminf(a, b), c), 0.f) + fminf(fmaxf(fmaxf(a, b), c), 0.f);
}
template <typename T>
__device__ __forceinline__ T minmod_slope(T l, T c, T r, T theta) {
  const T fwd = r - c;
  const T bwd = c - l;
  const T central = (fwd + bwd) * (T)0.5;  // x/2.0 == x*0.5 exactly in binary IEEE
  return minmod<T>(theta * fwd, central, theta * bwd);
}

// Half the minmod slope in Float64, minmod_slope's value times 0.5 bit for bit.
// Rounding is monotone, so the smaller of theta*fwd and theta*bwd is theta
// times the smaller difference: one product instead of two, and the halves and
// the choice among operands of one sign (the smaller magnitude has the smaller
// bits) are integer work. 4 FP64 instructions instead of 7.
__device__ __forceinline__ double half_slope(double l, double c, double r, double theta) {
  const double fwd = r - c, bwd = c - l;
  const double mean = exact::half(fwd + bwd);
  const unsigned long long bf = exact::bits(fwd), bb = exact::bits(bwd), bm = exact::bits(mean);
  const double t = theta * exact::from_bits(bf < bb ? bf : bb);
  const unsigned long long bt = exact::bits(t);
  const bool one_sign = (long long)((bf ^ bb) | (bt ^ bm) | (bf ^ bm)) >= 0;  // all four alike
  // with one sign, the smaller of t and mean is a zero when any of the four is
  const double s = exact::from_bits(bt < bm ? bt : bm);
  return one_sign && !exact::zero(s) ? exact::half(s) : 0.0;
}

// Practical-SWE linear reconstruction of one cell along one direction,
// src/reconstruction/linearreconstruction.jl:73-100. Inputs are (w, hu, hv) at
// the left, middle and right cells; outputs are face (h, hu, hv).
template <typename T>
__device__ __forceinline__ void reconstruct_cell(const Phys<T>& p, const T l[3], const T c[3], const T r[3], T Bl, T Br,
                                                 T L[3], T R[3]) {
  using A = Arith<T>;
  if constexpr (std::is_same<T, double>::value) {
    // The same values with half slopes: 0.5 * (2 (w - Bl)) is w - Bl.
    const double w = c[0];
    const double h0 = half_slope(l[0], w, r[0], p.theta);
    double wl = w - h0, wr = w + h0;
    const bool below_l = A::lt(wl, Bl);
    if (below_l || A::lt(wr, Br)) {
      const double d = below_l ? w - Bl : Br - w;
      wl = w - d;
      wr = w + d;
    }
    L[0] = wl - Bl;
    R[0] = wr - Br;
#pragma unroll
    for (int k = 1; k < 3; ++k) {
      const double hs = half_slope(l[k], c[k], r[k], p.theta);
      L[k] = c[k] - hs;
      R[k] = c[k] + hs;
    }
    return;
  }
  T s0 = minmod_slope<T>(l[0], c[0], r[0], p.theta);
  const T s1 = minmod_slope<T>(l[1], c[1], r[1], p.theta);
  const T s2 = minmod_slope<T>(l[2], c[2], r[2], p.theta);
  const T w = c[0];
  if (A::lt(w - (T)0.5 * s0, Bl)) {
    s0 = (T)2 * (w - Bl);
  } else if (A::lt(w + (T)0.5 * s0, Br)) {
    s0 = (T)2 * (Br - w);
  }
  L[0] = (c[0] - (T)0.5 * s0) - Bl;
  R[0] = (c[0] + (T)0.5 * s0) - Br;
  L[1] = c[1] - (T)0.5 * s1;
  R[1] = c[1] + (T)0.5 * s1;
  L[2] = c[2] - (T)0.5 * s2;
  R[2] = c[2] + (T)0.5 * s2;
}

// Friction factor of ImplicitFriction for a 2D cell, src/friction.jl:30-43,62-78:
// S = law(Cz, h*, |u|) with h* = desingularize(w - B_cell) and u = (hu, hv)/h*.
// When hu and hv are both zero, S is -0 and the implicit division is by 1:
// callers may skip it (friction_active).
template <typename T>
__device__ __forceinline__ bool friction_active(T hu, T hv) {
  return !(Arith<T>::is_zero(hu) && Arith<T>::is_zero(hv));
}
template <typename T>
__device__ __forceinline__ T friction_factor(const Phys<T>& p, T w, T hu, T hv, T Bc) {
  using A = Arith<T>;
  const T h = w - Bc;
  const T hs = desing<T>(h, p.kappa);
  T u, v;
  velocities<T>(p, h, hs, hu, hv, u, v);
  const T speed = A::sqrt_(u * u + v * v);
  T denom;
  if (p.friction == 1) {          // friction_bsa2012
    denom = vcbrt<T>(hs) * hs;
  } else if (p.friction == 2) {   // friction_fcg2016
    denom = vcbrt<T>(hs) * hs * hs;
  } else {                        // friction_bh2021
    denom = hs * hs;
  }
  return A::div(-p.Cz * speed, denom);
}

// out[1:2] ./= (1 - dt*S) (src/friction.jl:77); skipped when S is zero, where
// the division is by exactly 1.
template <typename T>
__device__ __forceinline__ void apply_friction(T tdt, T S, T& hu, T& hv) {
  using A = Arith<T>;
  if constexpr (sizeof(T) == 4) {  // a select instead of a branch
    const T f = A::is_zero(S) ? (T)1 : A::rcp((T)1 - tdt * S);
    hu = hu * f;
    hv = hv * f;
    return;
  }
  if (A::is_zero(S)) return;
  const T den = (T)1 - tdt * S;
  const typename A::Recip R = A::recip(den);
  hu = A::div_by(R, hu);
  hv = A::div_by(R, hv);
}

// Dry-cell clamp, src/timestepper/timestepper.jl:41-51.
template <typename T>
__device__ __forceinline__ void dry_clamp(const Phys<T>& p, T& w, T& hu, T& hv, T Bc) {
  using A = Arith<T>;
  if (A::lt(w - Bc, p.cutoff)) {
    w = A::max(w, Bc);
    hu = (T)0;
    hv = (T)0;
  }
}

}  // namespace vf
