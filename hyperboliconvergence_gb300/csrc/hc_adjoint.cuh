// hc_adjoint.cuh -- hand-written reverse-mode (discrete adjoint) versions of
// the pointwise functions of the residual path.  Each *_adj function takes the
// primal inputs, recomputes what it needs, and accumulates input adjoints from
// output adjoints (x_bar += (dy/dx)^T y_bar).  Branches (limiters, entropy fix,
// upwind switches) are differentiated along the branch the primal takes.
// The spectral-radius outputs are not differentiated: the adjoint treats the
// timestep of every step as a constant (frozen-timestep adjoint).
#pragma once

#include "hc_physics.cuh"

namespace hc {

template <class R> __host__ __device__ __forceinline__ R sgn(R x) { return x > R(0) ? R(1) : (x < R(0) ? R(-1) : R(0)); }

// primitive state adjoint: (u2, a2, h) -> (u, v, r, p); p and r also pass through
template <class R> struct StBar { R u, v, r, p, u2, a2, h; };

// (ir = 1/r given)
template <class R> __host__ __device__ __forceinline__ void prim_state_adj_ir(const Gas<R>& g, const R* q, R ir,
                                                                              StBar<R>& sb, R* qbar) {
  // h = a2*gamma1 + 0.5*u2
  sb.a2 += g.gamma1 * sb.h;
  sb.u2 += R(0.5) * sb.h;
  // u2 = u*u + v*v
  sb.u += R(2) * q[0] * sb.u2;
  sb.v += R(2) * q[1] * sb.u2;
  // a2 = gamma*R*t, t = p/(r*R): d a2/dp = gamma/r, d a2/dr = -gamma p/r^2
  const R gb = g.gamma * ir * sb.a2;
  sb.p += gb;
  sb.r -= gb * (q[3] * ir);
  qbar[0] += sb.u;
  qbar[1] += sb.v;
  qbar[2] += sb.r;
  qbar[3] += sb.p;
}
// exact flux adjoint, accumulating into the state adjoint of one side
template <class R> __host__ __device__ __forceinline__ void exact_flux_adj(R nx, R ny, const St<R>& s, const R* fbar,
                                                                  StBar<R>& sb) {
  const R un = nx * s.u + ny * s.v;
  const R mn = s.r * un;
  const R mnbar = s.u * fbar[0] + s.v * fbar[1] + fbar[2] + s.h * fbar[3];
  sb.u += mn * fbar[0];
  sb.v += mn * fbar[1];
  sb.p += nx * fbar[0] + ny * fbar[1];
  sb.h += mn * fbar[3];
  sb.r += un * mnbar;
  const R unbar = s.r * mnbar;
  sb.u += nx * unbar;
  sb.v += ny * unbar;
}

// Harten entropy fix of one nonlinear wave (roe.ipp:66-75) reversed
template <class R> __host__ __device__ __forceinline__ void entropy_fix_adj(R la, R ll, R lr, R lbar, R* labar, R* llbar,
                                                                   R* lrbar) {
  const R d1 = la - ll, d2 = lr - la;
  const R mx = fmax(d1, d2);
  const R le = R(0.05) * fmax(R(0), mx);
  const R laa = fabs(la);
  R laabar, lebar = R(0);
  if (laa > le) {
    laabar = lbar;
  } else if (le > R(0)) {
    lebar = R(0.5) * (R(1) - laa * laa / (le * le)) * lbar;
    laabar = (laa / le) * lbar;
  } else {
    laabar = R(0);  // exactly sonic, no expansion: the speed is 0 (roe_flux)
  }
  *labar += sgn(la) * laabar;
  if (mx > R(0)) {
    const R mbar = R(0.05) * lebar;
    if (d1 >= d2) { *labar += mbar; *llbar -= mbar; }
    else { *lrbar += mbar; *labar -= mbar; }
  }
}

// v with the sign of s, 0 where s is 0: v sgn(s) without an FP64 comparison
template <class R> __host__ __device__ __forceinline__ R times_sgn(R v, R s) { return sgn(s) * v; }
template <> __host__ __device__ __forceinline__ double times_sgn<double>(double v, double s) {
  const long long b = f64_bits(s);
  return (b << 1) == 0 ? 0.0 : (b < 0 ? -v : v);
}

// Reverse of roe_flux (hc_physics.cuh) for the four conserved flux components, with respect to
// the two primitive face states.  It reverses the multiplied-out form of the flux, in which the
// averaged density appears only through the averaging weight, and takes the sound speeds of the
// two states only where Harten's fix may act: 230 FP64 instructions with the forward values,
// against 330 for the transforms one by one.
template <class R>
__host__ __device__ __forceinline__ void roe_flux_adj(const Gas<R>& g, R nx, R ny, R A, const R* ql, const R* qr,
                                             const R* Fbar, R* qlbar, R* qrbar) {
  St<R> l, r;
  basis_state2(g, ql, qr, false, l, r);
  // ---- forward values
  const R unl = proj(nx, ny, l), unr = proj(nx, ny, r);
  R cr;
  sqrt_fast(r.r * l.ir, cr);
  const R wl = rcp_fast(R(1) + cr);
  const R wr = R(1) - wl;
  const R ua = mad(wl, l.u, wr * r.u);
  const R va = mad(wl, l.v, wr * r.v);
  const R ka = R(0.5) * mad(va, va, ua * ua);
  const R ha = mad(wl, l.h, wr * r.h);
  R aa, a1;
  sqrt_rcp(g.gm1 * (ha - ka), aa, a1);
  const R una = mad(nx, ua, ny * va);
  const R la1 = una - aa, la2 = una + aa;
  const R lam0 = fabs(una);
  R h1 = R(0.5) * fabs(la1), h2 = R(0.5) * fabs(la2);
  const bool near_fix = harten_near(unl, unr, l.a2, r.a2, una, aa);
  R al = R(0), ar = R(0), ial = R(0), iar = R(0);
  if (near_fix) {
    sqrt_rcp(l.a2, al, ial);
    sqrt_rcp(r.a2, ar, iar);
    auto fix = [](R la, R ll, R lr, R h) {
      const R le = R(0.05) * fmax(R(0), fmax(la - ll, lr - la));
      const R laa = fabs(la);
      return (laa > le || !(le > R(0))) ? h : R(0.25) * (le + laa * laa / le);
    };
    h1 = fix(la1, unl - al, unr - ar, h1);
    h2 = fix(la2, unl + al, unr + ar, h2);
  }
  const R d0 = mad(r.r, r.u, -(l.r * l.u));
  const R d1 = mad(r.r, r.v, -(l.r * l.v));
  const R d2 = r.r - l.r;
  const R d3 = mad(r.r, r.h, -r.p) - mad(l.r, l.h, -l.p);
  const R c0 = mad(nx, d0, ny * d1);
  const R c1 = mad(nx, d1, -(ny * d0));
  const R dp = g.gm1 * mad(-va, c1, mad(-ua, c0, mad(ka, d2, d3)));
  const R cn = mad(-ua, d2, c0), da = dp * a1;
  const R m1 = cn - da, m2 = cn + da;
  const R w1 = h1 * m1, w2 = h2 * m2;
  const R a12 = a1 * a1;
  const R z = mad(dp, a12, -d2);
  const R sm = w1 + w2, df = w2 - w1;
  const R drr = mad(-lam0, z, df * a1);
  const R t = mad(-va, d2, c1);
  const R sh = lam0 * t;
  // ---- reverse: G the adjoint of the central sums, -G of the dissipation's
  const R hA = R(0.5) * A;
  const R G0 = hA * Fbar[0], G1 = hA * Fbar[1], G2 = hA * Fbar[2], G3 = hA * Fbar[3];
  const R pn = mad(nx, G0, ny * G1);
  const R e0b = -pn, e1b = mad(ny, G0, -(nx * G1)), e3b = -G3;
  const R dppb = g.gamma1 * e3b;
  const R smb = mad(ua, e3b, e0b);
  const R shb = mad(va, e3b, e1b);
  const R drrb = mad(ua, e0b, mad(va, e1b, mad(ka, e3b, -G2)));
  R uab = mad(drr, e0b, sm * e3b);
  R vab = mad(drr, e1b, sh * e3b);
  R kab = drr * e3b;
  // the waves
  const R lam0b = mad(t, shb, -(z * drrb));
  const R tb = lam0 * shb, zb = -(lam0 * drrb);
  const R dfb = mad(a1, drrb, aa * dppb);
  R aab = df * dppb;
  R a1b = df * drrb;
  const R w1b = smb - dfb, w2b = smb + dfb;
  const R m1b = h1 * w1b, m2b = h2 * w2b;
  const R lam1b = R(0.5) * (m1 * w1b), lam2b = R(0.5) * (m2 * w2b);
  const R cnb = m1b + m2b, dab = m2b - m1b;
  const R dpb = mad(a12, zb, a1 * dab);
  a1b = mad(R(2) * da, zb, mad(dp, dab, a1b));
  // the pressure jump and the jumps in the face frame
  const R q = g.gm1 * dpb;
  kab = mad(d2, q, kab);
  uab = mad(-d2, cnb, mad(-c0, q, uab));
  vab = mad(-d2, tb, mad(-c1, q, vab));
  const R c0b = mad(-ua, q, cnb), c1b = mad(-va, q, tb);
  const R d2b = mad(ka, q, mad(-ua, cnb, mad(-va, tb, -zb)));
  const R d0b = mad(nx, c0b, -(ny * c1b));
  const R d1b = mad(ny, c0b, nx * c1b);
  // wave speeds
  R unab, unlb = R(0), unrb = R(0), la2l = R(0), la2r = R(0);
  {
    R la1b = R(0), la2b = R(0);
    if (near_fix) {
      R ll1b = R(0), lr1b = R(0), ll2b = R(0), lr2b = R(0);
      entropy_fix_adj(la1, unl - al, unr - ar, lam1b, &la1b, &ll1b, &lr1b);
      entropy_fix_adj(la2, unl + al, unr + ar, lam2b, &la2b, &ll2b, &lr2b);
      unlb = ll1b + ll2b;
      unrb = lr1b + lr2b;
      la2l = (ll2b - ll1b) * (R(0.5) * ial);
      la2r = (lr2b - lr1b) * (R(0.5) * iar);
    } else {
      la1b = times_sgn(lam1b, la1);
      la2b = times_sgn(lam2b, la2);
    }
    unab = times_sgn(lam0b, una) + (la1b + la2b);
    aab = mad(-a12, a1b, aab) + (la2b - la1b);
  }
  uab = mad(nx, unab, uab);
  vab = mad(ny, unab, vab);
  const R hab = (R(0.5) * g.gm1) * (a1 * aab);
  kab = kab - hab;
  uab = mad(ua, kab, uab);
  vab = mad(va, kab, vab);
  // the averaging weight
  const R wlb = mad(l.h - r.h, hab, mad(l.u - r.u, uab, (l.v - r.v) * vab));
  const R k = (R(-0.5) * cr) * ((wl * wl) * wlb);
  // the two states: jumps, averages and central fluxes
  auto side = [&](const St<R>& s, const R* qs, R un, R w, R sg, R unb, R a2x, R* qbar) {
    const R mnb = mad(s.u, G0, mad(s.v, G1, mad(s.h, G3, G2)));
    const R ub = mad(s.r, mad(nx, mnb, mad(un, G0, sg * d0b)), mad(nx, unb, w * uab));
    const R vb = mad(s.r, mad(ny, mnb, mad(un, G1, sg * d1b)), mad(ny, unb, w * vab));
    const R hb = mad(s.r, mad(un, G3, sg * q), w * hab);
    const R rb = mad(un, mnb, sg * mad(s.u, d0b, mad(s.v, d1b, mad(s.h, q, mad(k, s.ir, d2b)))));
    // primitive -> state (prim_state_adj)
    const R gb = (g.gamma * s.ir) * mad(g.gamma1, hb, a2x);
    qbar[0] += mad(qs[0], hb, ub);
    qbar[1] += mad(qs[1], hb, vb);
    qbar[2] += mad(-gb, qs[3] * s.ir, rb);
    qbar[3] += gb + mad(-sg, q, pn);
  };
  side(l, ql, unl, wl, R(-1), unlb, la2l, qlbar);
  side(r, qr, unr, wr, R(1), unrb, la2r, qrbar);
}

// Reverse of rusanov_flux (conservationLaws/base/fluxes/rusanovFlux.ipp:2-50)
template <class R>
__host__ __device__ __forceinline__ void rusanov_flux_adj(const Gas<R>& g, R nx, R ny, R A, const R* ql, const R* qr,
                                                 const R* Fbar, R* qlbar, R* qrbar) {
  St<R> l, r;
  basis_state2(g, ql, qr, false, l, r);
  const R unl = proj(nx, ny, l), unr = proj(nx, ny, r);
  R al, ar;
  sqrt_fast(l.a2, al);
  sqrt_fast(r.a2, ar);
  const R srl = fabs(unl) + al, srr = fabs(unr) + ar;
  const R lambda = fmax(srl, srr);
  const R s = R(-0.5) * (lambda * A);
  const R dc[4] = {r.r * r.u - l.r * l.u, r.r * r.v - l.r * l.v, r.r - l.r, (r.r * r.h - r.p) - (l.r * l.h - l.p)};
  StBar<R> lb{}, rb{};
  // dissipation s*dc
  R sb = R(0);
#pragma unroll
  for (int i = 0; i < 4; ++i) sb += dc[i] * Fbar[i];
  const R lamb = R(-0.5) * A * sb;
  rb.r += r.u * s * Fbar[0]; rb.u += r.r * s * Fbar[0]; lb.r -= l.u * s * Fbar[0]; lb.u -= l.r * s * Fbar[0];
  rb.r += r.v * s * Fbar[1]; rb.v += r.r * s * Fbar[1]; lb.r -= l.v * s * Fbar[1]; lb.v -= l.r * s * Fbar[1];
  rb.r += s * Fbar[2]; lb.r -= s * Fbar[2];
  rb.r += r.h * s * Fbar[3]; rb.h += r.r * s * Fbar[3]; rb.p -= s * Fbar[3];
  lb.r -= l.h * s * Fbar[3]; lb.h -= l.r * s * Fbar[3]; lb.p += s * Fbar[3];
  if (srl >= srr) {
    lb.u += nx * sgn(unl) * lamb; lb.v += ny * sgn(unl) * lamb; lb.a2 += div_fast(lamb, R(2) * al);
  } else {
    rb.u += nx * sgn(unr) * lamb; rb.v += ny * sgn(unr) * lamb; rb.a2 += div_fast(lamb, R(2) * ar);
  }
  R fe[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) fe[i] = R(0.5) * A * Fbar[i];
  exact_flux_adj(nx, ny, l, fe, lb);
  exact_flux_adj(nx, ny, r, fe, rb);
  prim_state_adj_ir(g, ql, l.ir, lb, qlbar);
  prim_state_adj_ir(g, qr, r.ir, rb, qrbar);
}

// van Albada's value z = ab(a+b)/(a^2+b^2+tiny) and its derivatives along the taken branch
// for four (a, b) pairs, FP64, 17 instructions each: 0 with zero derivatives where a b < 0 or
// a = b = 0 (the formula's own derivatives there).  The sign and range tests read the bits on
// the integer pipe.
__host__ __device__ __forceinline__ void vanalbada_vg4(const double* a, const double* b, double* z, double* da,
                                                       double* db) {
#pragma unroll
  for (int v = 0; v < 4; ++v) {
    const double ab = a[v] * b[v];
    const long long bits = f64_bits(ab);
    const unsigned long long mag = (unsigned long long)bits << 1;  // magnitude bits
    // not (a b < 0): a b is +0, -0, positive or NaN (which propagates); and not a = b = 0
    const bool both_zero = ((unsigned long long)f64_bits(a[v]) << 1) == 0 && ((unsigned long long)f64_bits(b[v]) << 1) == 0;
    const bool on = (bits >= 0 || mag == 0 || mag > (0x7ff0000000000000ULL << 1)) && !both_zero;
    if (!on) { z[v] = da[v] = db[v] = 0.0; continue; }
    const double a2 = a[v] * a[v], b2 = b[v] * b[v], den = a2 + b2;
    double iden;
#ifdef __CUDA_ARCH__
    if (f64_in_window(den)) iden = rcp_step(den);
    else
#endif
      iden = 1.0 / (den + Lim<double>::tiny());
    const double ab2 = ab + ab;
    const double zz = (ab * (a[v] + b[v])) * iden;
    z[v] = zz;
    da[v] = fma(-zz, a[v] + a[v], ab2 + b2) * iden;
    db[v] = fma(-zz, b[v] + b[v], a2 + ab2) * iden;
  }
}

// derivative of limit(kind, a, b) along the taken branch: *da, *db
template <class R> __host__ __device__ __forceinline__ void limit_grad(int kind, R a, R b, R* da, R* db) {
  const R tiny = Lim<R>::tiny();
  *da = R(0); *db = R(0);
  switch (kind) {
    case LIM_NOLIMIT1: return;
    case LIM_NOLIMIT2: *da = R(0.5); *db = R(0.5); return;
    case LIM_NOLIMIT3: *da = R(0.33333333333333333) * R(2); *db = R(0.33333333333333333); return;
    case LIM_VANALBADA: {
      if (a * b < R(0)) return;
      // z = num/den; dz = (dnum - z*dden)/den (no den^2: it underflows at a = b = 0)
      const R num = b * (a * a) + a * (b * b), den = a * a + b * b + tiny;
      const R iden = rcp_near(den);
      const R z = num * iden;
      *da = ((R(2) * a * b + b * b) - z * R(2) * a) * iden;
      *db = ((a * a + R(2) * a * b) - z * R(2) * b) * iden;
      return;
    }
    case LIM_MINMOD:
      if (a > R(0)) { if (a <= fmax(b, R(0))) *da = R(1); else if (b > R(0)) *db = R(1); }
      else { if (a >= fmin(b, R(0))) *da = R(1); else if (b < R(0)) *db = R(1); }
      return;
    case LIM_VANLEER: {
      const R num = a * fabs(b) + fabs(a) * b, den = fabs(a) + fabs(b) + tiny;
      const R iden = rcp_near(den);
      const R z = num * iden;
      *da = ((fabs(b) + sgn(a) * b) - z * sgn(a)) * iden;
      *db = ((a * sgn(b) + fabs(a)) - z * sgn(b)) * iden;
      return;
    }
    default: return;  // other limiters are not differentiated
  }
}

// Jacobian transposes of the primitive <-> conserved maps (the RK update
// cons(q0) + R*f -> prim): prim adjoint at state q -> conserved adjoint, and
// conserved adjoint at state q0 -> prim adjoint.
// (one reciprocal of the density and the gas's 1/(gamma-1) instead of four divisions: the
// reverse passes are bound by the FP64 pipe)
template <class R> __host__ __device__ __forceinline__ void cons2prim_adj(const Gas<R>& g, const R* q, const R* pb, R* cb) {
  const R u = q[0], v = q[1], ir = rcp_near(q[2]);
  cb[0] = pb[0] * ir - g.gm1 * u * pb[3];
  cb[1] = pb[1] * ir - g.gm1 * v * pb[3];
  cb[2] = pb[2] - (u * pb[0] + v * pb[1]) * ir + R(0.5) * g.gm1 * (u * u + v * v) * pb[3];
  cb[3] = g.gm1 * pb[3];
}
template <class R> __host__ __device__ __forceinline__ void prim2cons_adj(const Gas<R>& g, const R* q, const R* cb, R* pb) {
  const R u = q[0], v = q[1], r = q[2];
  pb[0] += r * cb[0] + r * u * cb[3];
  pb[1] += r * cb[1] + r * v * cb[3];
  pb[2] += u * cb[0] + v * cb[1] + cb[2] + R(0.5) * (u * u + v * v) * cb[3];
  pb[3] += cb[3] * g.gamma1;
}

}  // namespace hc
