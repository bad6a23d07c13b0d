// hc_pair.cuh -- pairs of FP32 values: one instruction (FFMA2 and its kin) computes both.  It has
// the rate of two FP32 instructions but takes one issue slot, and issue is what bounds the FP32
// and the double-float stage.  Each half rounds as the scalar instruction does.
#pragma once

#include "hc_physics.cuh"

namespace hc {

struct f2 { unsigned long long v; };
__device__ __forceinline__ f2 pair(float lo, float hi) {
  f2 r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r.v) : "f"(lo), "f"(hi));
  return r;
}
__device__ __forceinline__ float lo(f2 a) {
  float x, y;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(x), "=f"(y) : "l"(a.v));
  return x;
}
__device__ __forceinline__ float hi(f2 a) {
  float x, y;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(x), "=f"(y) : "l"(a.v));
  return y;
}
__device__ __forceinline__ f2 fma2(f2 a, f2 b, f2 c) {
  f2 r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r.v) : "l"(a.v), "l"(b.v), "l"(c.v));
  return r;
}
__device__ __forceinline__ f2 mul2(f2 a, f2 b) {
  f2 r;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v));
  return r;
}
__device__ __forceinline__ f2 add2(f2 a, f2 b) {
  f2 r;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v));
  return r;
}
__device__ __forceinline__ f2 pair(float x) { return pair(x, x); }
__device__ __forceinline__ f2 neg2(f2 a) { return mul2(a, pair(-1.f)); }
__device__ __forceinline__ f2 sub2(f2 a, f2 b) { return fma2(b, pair(-1.f), a); }

// ---- pairs of double-float values, operation by operation as hc_df64.cuh has them (the same bits)
struct df2 { f2 hi, lo; };
__device__ __forceinline__ df2 pair(df64 x, df64 y) { return {pair(x.hi, y.hi), pair(x.lo, y.lo)}; }
__device__ __forceinline__ df2 pair(df64 x) { return pair(x, x); }
__device__ __forceinline__ df64 lo(df2 a) { return df64(lo(a.hi), lo(a.lo)); }
__device__ __forceinline__ df64 hi(df2 a) { return df64(hi(a.hi), hi(a.lo)); }
__device__ __forceinline__ df2 two_sum2(f2 a, f2 b) {
  const f2 s = add2(a, b), bb = sub2(s, a);
  return {s, add2(sub2(a, sub2(s, bb)), sub2(b, bb))};
}
__device__ __forceinline__ df2 fast_two_sum2(f2 a, f2 b) {
  const f2 s = add2(a, b);
  return {s, sub2(b, sub2(s, a))};
}
__device__ __forceinline__ df2 operator+(df2 a, df2 b) {
  const df2 s = two_sum2(a.hi, b.hi);
  return fast_two_sum2(s.hi, add2(s.lo, add2(a.lo, b.lo)));
}
__device__ __forceinline__ df2 operator-(df2 a, df2 b) {
  const f2 s = sub2(a.hi, b.hi), bb = sub2(s, a.hi);
  const f2 e = sub2(sub2(a.hi, sub2(s, bb)), add2(b.hi, bb));
  return fast_two_sum2(s, add2(e, sub2(a.lo, b.lo)));
}
__device__ __forceinline__ df2 operator*(df2 a, df2 b) {
  const f2 p = mul2(a.hi, b.hi), np = neg2(p);
  const f2 e = fma2(a.lo, b.hi, fma2(a.hi, b.lo, fma2(a.hi, b.hi, np)));
  const f2 s = add2(p, e);
  return {s, sub2(e, add2(s, np))};
}
__device__ __forceinline__ df2 quotient2(df2 a, df2 b, f2 rb, f2 q1) {
  const f2 n1 = neg2(q1);
  const df2 r = two_sum2(fma2(n1, b.hi, a.hi), fma2(n1, b.lo, a.lo));
  const f2 q2 = mul2(r.hi, rb), n2 = neg2(q2);
  const f2 e = add2(fma2(n2, b.hi, r.hi), fma2(n2, b.lo, r.lo));
  return fast_two_sum2(q1, fma2(e, rb, q2));
}
__device__ __forceinline__ f2 near_rcp2(f2 b) { return pair(dd::near_rcp(lo(b)), dd::near_rcp(hi(b))); }
__device__ __forceinline__ df2 operator/(df2 a, df2 b) {
  const f2 rb = near_rcp2(b.hi), q0 = mul2(a.hi, rb);
  return quotient2(a, b, rb, fma2(fma2(neg2(q0), b.hi, a.hi), rb, q0));
}
__device__ __forceinline__ df2 rcp(df2 b) {
  const f2 rb = near_rcp2(b.hi);
  return quotient2({pair(1.f), pair(0.f)}, b, rb, rb);
}
__device__ __forceinline__ df2 half(df2 a) { return {mul2(a.hi, pair(0.5f)), mul2(a.lo, pair(0.5f))}; }

// the limiter of two sides with the same central difference (limit<df64>)
__device__ __forceinline__ df2 limit2(int kind, df64 a, df2 b) {
  if (kind == LIM_VANALBADA) {
    const df2 aa = pair(a), ab = aa * b;
    df2 d = pair(a * a) + b * b;
    d.hi = pair(fmaxf(lo(d.hi), FLT_MIN), fmaxf(hi(d.hi), FLT_MIN));
    const df2 s = ab * (aa + b) / d;
    return pair(lo(ab.hi) < 0.f ? df64() : lo(s), hi(ab.hi) < 0.f ? df64() : hi(s));
  }
  if (kind == LIM_VANLEER) {
    const df2 aa = pair(a), ab = aa * b;
    const df2 s = (ab + ab) / (aa + b);
    return pair(lo(ab.hi) <= 0.f ? df64() : lo(s), hi(ab.hi) <= 0.f ? df64() : hi(s));
  }
  return pair(limit<df64>(kind, a, lo(b)), limit<df64>(kind, a, hi(b)));
}
// the two states of a face from the pairs {left, right} of its primitive values (prim_state_ir)
__device__ __forceinline__ void prim_states(const Gas<df64>& g, const df2* q, St<df64>& l, St<df64>& r) {
  const df2 ir = rcp(q[2]);
  const df2 u2 = q[1] * q[1] + q[0] * q[0];
  const df2 a2 = pair(g.gamma) * (q[3] * ir);
  const df2 h = a2 * pair(g.gamma1) + half(u2);
  l.u = lo(q[0]); l.v = lo(q[1]); l.r = lo(q[2]); l.p = lo(q[3]);
  l.u2 = lo(u2); l.ir = lo(ir); l.a2 = lo(a2); l.h = lo(h);
  r.u = hi(q[0]); r.v = hi(q[1]); r.r = hi(q[2]); r.p = hi(q[3]);
  r.u2 = hi(u2); r.ir = hi(ir); r.a2 = hi(a2); r.h = hi(h);
}

}  // namespace hc
