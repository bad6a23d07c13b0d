// hc_df64.cuh -- double-float arithmetic: a value is the unevaluated sum
// hi + lo of two FP32 numbers with |lo| <= ulp(hi)/2, giving a ~48-bit
// significand (relative rounding ~2^-47) computed entirely on the FP32 pipes.
//
// Algorithms: error-free transformations of Knuth (TwoSum, TAOCP vol. 2,
// 4.2.2) and Dekker ("A floating-point technique for extending the available
// precision", Numer. Math. 18, 1971; Fast2Sum), products through the fused
// multiply-add (the residual a*b - fl(a*b) is one FMA), division and square root by
// the remainder of an FP32 quotient or root, exact in one FMA (after Karp & Markstein,
// "High-precision division and square root", ACM TOMS 23(4), 1997).  The exponent range is FP32's.
//
// Written for __host__ and __device__ so the same code is testable on a CPU.
// The type and its functions live in hc::dd and are found by argument-dependent
// lookup, so code in namespace hc keeps calling the global sqrt/fabs/fmax for
// double and float.
#pragma once

#include <cfloat>
#include <cmath>
#include <cuda_runtime.h>

namespace hc {
namespace dd {

struct df64 {
  float hi, lo;
  __host__ __device__ constexpr df64() : hi(0.f), lo(0.f) {}
  __host__ __device__ constexpr df64(float h, float l) : hi(h), lo(l) {}
  // split of a double: hi = rn(x), lo = rn(x - hi); exact for |x| in FP32 range
  __host__ __device__ constexpr df64(double x) : hi(float(x)), lo(float(x - double(float(x)))) {}
  __host__ __device__ constexpr df64(int x) : df64(double(x)) {}
  __host__ __device__ double to_double() const { return double(hi) + double(lo); }
};

__host__ __device__ __forceinline__ float df_fma(float a, float b, float c) {
#ifdef __CUDA_ARCH__
  return __fmaf_rn(a, b, c);
#else
  return std::fma(a, b, c);
#endif
}

// s + e == a + b exactly (Knuth)
__host__ __device__ __forceinline__ df64 two_sum(float a, float b) {
  const float s = a + b;
  const float bb = s - a;
  const float e = (a - (s - bb)) + (b - bb);
  return df64(s, e);
}
// s + e == a + b exactly when |a| >= |b| (Dekker)
__host__ __device__ __forceinline__ df64 fast_two_sum(float a, float b) {
  const float s = a + b;
  const float e = b - (s - a);
  return df64(s, e);
}

// One TwoSum on the high parts, the low parts added in FP32: the error is bounded
// by ~2^-47 (|a| + |b|), relative to the operands rather than to the sum (the
// form with a second TwoSum on the low parts is relative to the sum but costs
// twice the instructions; no quantity of the stage needs more than
// operand-relative accuracy in a difference).
__host__ __device__ __forceinline__ df64 operator+(df64 a, df64 b) {
  const df64 s = two_sum(a.hi, b.hi);
  return fast_two_sum(s.hi, s.lo + (a.lo + b.lo));
}
__host__ __device__ __forceinline__ df64 operator-(df64 a) { return df64(-a.hi, -a.lo); }
__host__ __device__ __forceinline__ df64 operator-(df64 a, df64 b) { return a + (-b); }
__host__ __device__ __forceinline__ df64 operator*(df64 a, df64 b) {
  const float p = a.hi * b.hi;
  float e = df_fma(a.hi, b.hi, -p);
  e = df_fma(a.hi, b.lo, e);
  e = df_fma(a.lo, b.hi, e);
  return fast_two_sum(p, e);
}
__host__ __device__ __forceinline__ df64 mul_f(df64 a, float b) {
  const float p = a.hi * b;
  float e = df_fma(a.hi, b, -p);
  e = df_fma(a.lo, b, e);
  return fast_two_sum(p, e);
}
// FP32 reciprocal estimate of b.hi from the approximate-reciprocal instruction
__host__ __device__ __forceinline__ float approx_rcp(float x) {
#ifdef __CUDA_ARCH__
  float r;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
#else
  return 1.0f / x;
#endif
}
// The reciprocal of b.hi: the estimate and one Newton step, within half a unit or so.
__host__ __device__ __forceinline__ float near_rcp(float bh) {
  // the approximate reciprocal flushes subnormal inputs and results: take it of
  // b.hi scaled by a power of two into range, then undo the scaling (exact)
  const float m = fabsf(bh);
  const float sc = m > 0x1p125f ? 0x1p-64f : (m < 0x1p-125f ? 0x1p64f : 1.0f);
  const float x = bh * sc, r = approx_rcp(x);
  return df_fma(r, df_fma(-x, r, 1.0f), r) * sc;
}
// Second part of a quotient from its FP32 value q1, right to a unit: the remainder
// a.hi - q1 b.hi is exact in one FMA, the low parts join it in a TwoSum, and the correction
// by it is itself corrected once.  Over 4 million quotients (exponents within 9) the largest
// error is 2^-46.2, the rms 2^-49.3 (reciprocals 2^-47.2, 2^-49.7), with the estimate
// disturbed by a unit; two remainders in double-float, as Karp & Markstein's scheme has them,
// make 2^-46.0 and 2^-49.1 (2^-46.1, 2^-49.3) for twice the instructions (50; these are 28).
__host__ __device__ __forceinline__ df64 quotient(df64 a, df64 b, float rb, float q1) {
  const df64 r = two_sum(df_fma(-q1, b.hi, a.hi), df_fma(-q1, b.lo, a.lo));
  const float q2 = r.hi * rb;
  const float e = df_fma(-q2, b.hi, r.hi) + df_fma(-q2, b.lo, r.lo);
  return fast_two_sum(q1, df_fma(e, rb, q2));
}
__host__ __device__ __forceinline__ df64 operator/(df64 a, df64 b) {
  const float rb = near_rcp(b.hi);
  const float q0 = a.hi * rb;
  return quotient(a, b, rb, df_fma(df_fma(-q0, b.hi, a.hi), rb, q0));
}
__host__ __device__ __forceinline__ df64 rcp(df64 b) {
  const float rb = near_rcp(b.hi);
  return quotient(df64(1.0f, 0.0f), b, rb, rb);
}
// exact
__host__ __device__ __forceinline__ df64 half(df64 a) { return df64(0.5f * a.hi, 0.5f * a.lo); }
__host__ __device__ __forceinline__ df64& operator+=(df64& a, df64 b) { return a = a + b; }
__host__ __device__ __forceinline__ df64& operator-=(df64& a, df64 b) { return a = a - b; }
__host__ __device__ __forceinline__ df64& operator*=(df64& a, df64 b) { return a = a * b; }

__host__ __device__ __forceinline__ bool operator<(df64 a, df64 b) { return a.hi < b.hi || (a.hi == b.hi && a.lo < b.lo); }
__host__ __device__ __forceinline__ bool operator>(df64 a, df64 b) { return b < a; }
__host__ __device__ __forceinline__ bool operator<=(df64 a, df64 b) { return !(b < a); }
__host__ __device__ __forceinline__ bool operator>=(df64 a, df64 b) { return !(a < b); }
__host__ __device__ __forceinline__ bool operator==(df64 a, df64 b) { return a.hi == b.hi && a.lo == b.lo; }

__host__ __device__ __forceinline__ df64 fabs(df64 a) { return a.hi < 0.f ? -a : a; }
__host__ __device__ __forceinline__ df64 fmax(df64 a, df64 b) { return (a < b) ? b : a; }
__host__ __device__ __forceinline__ df64 fmin(df64 a, df64 b) { return (b < a) ? b : a; }
// Square root: from the approximate 1/sqrt(a.hi) the root and half its inverse, one coupled
// Newton step each and one more for the root, which then is right to a unit; the remainder
// a - s^2 (exact in one FMA) gives the second part.  Error 2^-46.2 at most, rms 2^-49.4, like
// the form on the correctly rounded root and a full division, in 12 instructions.  Outside
// the estimate's range that form.
__host__ __device__ __forceinline__ df64 sqrt(df64 a) {
#ifdef __CUDA_ARCH__
  if (a.hi > 0x1p-100f && a.hi < 0x1p100f) {
    float r;
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(a.hi));
    float s = a.hi * r, h = 0.5f * r;
    const float d = df_fma(-s, h, 0.5f);
    s = df_fma(s, d, s);
    h = df_fma(h, d, h);
    s = df_fma(df_fma(-s, s, a.hi), h, s);
    return fast_two_sum(s, (df_fma(-s, s, a.hi) + a.lo) * h);
  }
#endif
  if (!(a.hi > 0.f)) return df64(a.hi == 0.f ? 0.f : NAN, 0.f);
  const float s = sqrtf(a.hi);
  const float p = s * s;
  const float pe = df_fma(s, s, -p);
  const float e = ((a.hi - p) - pe + a.lo) * (0.5f / s);
  return fast_two_sum(s, e);
}

#ifdef __CUDACC__
// The split of a double without the FP64 pipe, whose two conversions, difference and second
// conversion back take 67 cycles of it per warp: the high word's bits shifted into an FP32 value
// and rounded by hand (to nearest, ties to even), the rest of the mantissa as a signed integer
// times its unit.  Same result; small or large values take the conversions.
__device__ __forceinline__ df64 split(double x) {
  const unsigned h = unsigned(__double2hiint(x)), l = unsigned(__double2loint(x));
  const unsigned e = (h >> 20) & 0x7ffu;  // FP32 exponent field = e - 896
  if (e - (896u + 64u) >= 254u - 64u) return (h << 1 | l) == 0u ? df64() : df64(x);
  const unsigned sign = h & 0x80000000u;
  const unsigned t = __funnelshift_l(l, (h & 0x7fffffffu) - (896u << 20), 3);
  const unsigned rest = l & 0x1fffffffu;
  const unsigned up = rest + (t & 1u) > 0x10000000u ? 1u : 0u;
  const float unit = __uint_as_float(((e - 896u - 52u) << 23) | sign);
  return df64(__uint_as_float((t + up) | sign), float(int(rest) - int(up << 29)) * unit);
}
#endif
__host__ __device__ __forceinline__ bool isfinite(df64 a) { return ::isfinite(a.hi); }

}  // namespace dd
using dd::df64;
}  // namespace hc
