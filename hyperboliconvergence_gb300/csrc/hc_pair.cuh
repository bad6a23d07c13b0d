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
// The two states of a face from the pairs {left, right} of its primitive values (prim_state_ir).
struct StPair { df2 u, v, r, p, u2, ir, a2, h; };
__device__ __forceinline__ StPair prim_states(const Gas<df64>& g, const df2* q) {
  StPair s;
  s.u = q[0]; s.v = q[1]; s.r = q[2]; s.p = q[3];
  s.ir = rcp(s.r);
  s.u2 = s.v * s.v + s.u * s.u;
  s.a2 = pair(g.gamma) * (s.p * s.ir);
  s.h = s.a2 * pair(g.gamma1) + half(s.u2);
  return s;
}
__device__ __forceinline__ St<df64> left_state(const StPair& s) {
  St<df64> l;
  l.u = lo(s.u); l.v = lo(s.v); l.r = lo(s.r); l.p = lo(s.p);
  l.u2 = lo(s.u2); l.ir = lo(s.ir); l.a2 = lo(s.a2); l.h = lo(s.h);
  return l;
}
__device__ __forceinline__ St<df64> right_state(const StPair& s) {
  St<df64> r;
  r.u = hi(s.u); r.v = hi(s.v); r.r = hi(s.r); r.p = hi(s.p);
  r.u2 = hi(s.u2); r.ir = hi(s.ir); r.a2 = hi(s.a2); r.h = hi(s.h);
  return r;
}
__device__ __forceinline__ df64 sum(df2 a) { return lo(a) + hi(a); }

// roe_flux<df64> with its twins packed -- the two sides, the components of velocity, momentum and
// force, the two acoustic waves -- in the same operations, so with the same bits: about 620
// instructions instead of 930.  512 x 1024 O-grid, two steps: 1.64 -> 1.57 ms.
template <bool FACE>
__device__ __forceinline__ Flux5<df64> roe_flux_pairs(const Gas<df64>& g, df64 nx, df64 ny, df64 A, const StPair& s,
                                                      bool want_lam) {
  using R = df64;
  const df2 n = pair(nx, ny);
  const df2 un = pair(nx) * s.u + pair(ny) * s.v;
  const R unl = lo(un), unr = hi(un);
  R cr;
  sqrt_fast(hi(s.r) * lo(s.ir), cr);
  const R wl = rcp_fast(R(1) + cr);
  const R wr = R(1) - wl;
  const df2 ul = pair(lo(s.u), lo(s.v)), ur = pair(hi(s.u), hi(s.v));
  const df2 ua = pair(wl) * ul + pair(wr) * ur;  // the averaged velocity
  const R ka = half(sum(ua * ua));
  const R ha = sum(pair(wl, wr) * s.h);
  const R a2a = g.gm1 * (ha - ka);
  R aa, a1;
  sqrt_rcp(a2a, aa, a1);
  const R una = sum(n * ua);
  const df2 la = pair(una) + pair(-aa, aa);
  const R lam0 = fabs(una);
  R lam1 = fabs(lo(la)), lam2 = fabs(hi(la));
  Flux5<R> o;
  o.lam = R(0);
  const bool near_fix = harten_near(unl, unr, lo(s.a2), hi(s.a2), una, aa);
  if (want_lam || near_fix) {
    R al, ar;
    sqrt_fast(lo(s.a2), al);
    sqrt_fast(hi(s.a2), ar);
    if (near_fix) roe_entropy_fix(unl, unr, al, ar, lo(la), hi(la), lam1, lam2);
    o.lam = max_pos(max_pos(fabs(unl) + al, fabs(unr) + ar), lam0 + aa) * A;
  }
  const df2 mu = s.r * s.u, mv = s.r * s.v, me = s.r * s.h - s.p;
  const R d0 = hi(mu) - lo(mu), d1 = hi(mv) - lo(mv), d2 = hi(s.r) - lo(s.r), d3 = hi(me) - lo(me);
  const df2 c = pair(nx) * pair(d0, d1) + pair(ny) * pair(d1, -d0);
  const df2 x = FACE ? pair(una, nx * hi(ua) - ny * lo(ua)) : ua;
  const df2 xc = x * c;
  const R dp = g.gm1 * (((ka * d2 + d3) - lo(xc)) - hi(xc));
  const df2 cs = c - x * pair(d2);  // the normal and tangential momentum jumps about the average
  const R da = dp * a1;
  const df2 w = half(pair(lam1, lam2)) * (pair(lo(cs)) + pair(-da, da));
  const R z = dp * (a1 * a1) - d2;
  const df2 sd = pair(hi(w)) + pair(lo(w), -lo(w));
  const R sm = lo(sd);
  const df2 da2 = pair(hi(sd)) * pair(aa, a1);
  const R dpp = lo(da2);
  const R drr = hi(da2) - lam0 * z;
  const R sh = lam0 * hi(cs);
  const df2 e = x * pair(drr) + pair(sm, sh);
  const df2 m = s.r * un;
  const R hA = half(A);
  const df2 cu = m * s.u + s.p * pair(nx), cv = m * s.v + s.p * pair(ny), ch = m * s.h;
  const df2 ds = pair(ny, nx) * pair(hi(e)) + pair(-nx, ny) * pair(lo(e));
  const df2 f01 = pair(lo(cu), lo(cv)) + pair(hi(cu), hi(cv)) + pair(lo(ds), -hi(ds));
  const df2 xs = x * pair(sm, sh);
  const R f2 = sum(m) - drr;
  const R f3 = sum(ch) - (ka * drr + (hi(xs) + (lo(xs) + g.gamma1 * dpp)));
  const df2 oa = pair(hA) * f01, ob = pair(hA) * pair(f2, f3);
  o.f[0] = lo(oa); o.f[1] = hi(oa); o.f[2] = lo(ob); o.f[3] = hi(ob);
  return o;
}
template <int FK>
__device__ __forceinline__ Flux5<df64> face_flux_pairs(const Gas<df64>& g, df64 nx, df64 ny, df64 A, const StPair& s,
                                                       bool want_lam) {
  if constexpr (FK == FLUX_ROE) return roe_flux_pairs<false>(g, nx, ny, A, s, want_lam);
  else if constexpr (FK == FLUX_ROE_FACE) return roe_flux_pairs<true>(g, nx, ny, A, s, want_lam);
  else return face_flux<df64, FK>(g, nx, ny, A, left_state(s), right_state(s), want_lam);
}

}  // namespace hc
