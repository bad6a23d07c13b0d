// hc_oned.cuh -- the one-dimensional Euler path: one fused RK stage per launch over
// tiles of TB cells (interiorResidual in 1D, spatial/residualCalc.h:74-127, with the
// 1D boundary loops and LSQ metrics of spatial/boundary/*.h and spatial/lsqMetrics.h).
// State: 3 planes {u, rho, p}; residual: 3 flux planes {rho u, rho, rho E} + the
// spectral-radius sum.  The fluxes and far-field updates are the 2D device functions
// with the second velocity 0 and face normals (+-1, 0): the reference's nDim = 1
// instantiations compute the same (pinned by the golden vectors).
#pragma once

#include "hc_kernels.cuh"

namespace hc {

// per-face 1D records (nc + 1 faces, face f at node f between cells f-1 and f)
enum Face1Field { F1_DL = 0, F1_DR, F1_IDLR, F1_WL, F1_SL, F1_WR, F1_SR, F1_DX, F1_WW, F1REC };

template <class R> struct Stage1DArgs {
  int nc;
  int bc[2];
  Gas<R> gas;
  int limiter;
  const R* q;       // stage state (3 planes)
  const R* q0;      // state at the start of the step
  const R* rec;     // F1REC planes of nc + 1 face records
  const R* vol;
  const R* gref[2]; // reference values of sides 0 / 1 (3 values)
  R* res_out;       // 4 planes or null
  const R* res_prev[4];
  R alpha[4];
  int stage, mode;
  R beta, cfl;
  StepInfo* info;
  R* q_out;
  int norm_stage0;
};

// A warp takes 30 cells: lane l holds cell i0 - 1 + l, lanes 0 and 31 the neighbours' (with the
// cells beyond those in a second register), and the face on its left.  An SM's sub-partition
// starts one FP64 instruction per 64 cycles whatever the number of active lanes, so a line is
// as fast as its warps are spread: one warp per block and 30-cell tiles.
constexpr int kLineCells = 30;

template <class R> __device__ __forceinline__ St<R> st1(const Gas<R>& g, const R* q) {
  St<R> s;
  s.u = q[0]; s.v = R(0); s.r = q[1]; s.p = q[2];
  s.u2 = s.u * s.u;
  s.ir = rcp_fast(s.r);
  s.a2 = g.gamma * (s.p * s.ir);
  s.h = mad(s.a2, g.gamma1, R(0.5) * s.u2);
  return s;
}

// roe_flux on the line: velocity along the face normal (1, 0), the second one 0, area 1
template <class R> __device__ __forceinline__ Flux5<R> roe_flux_1d(const Gas<R>& g, const St<R>& l, const St<R>& r, bool want_lam) {
  R cr;
  sqrt_fast(r.r * l.ir, cr);
  const R wl = rcp_fast(R(1) + cr);
  const R wr = R(1) - wl;
  const R ua = mad(wl, l.u, wr * r.u);
  const R ka = R(0.5) * (ua * ua);
  const R ha = mad(wl, l.h, wr * r.h);
  R aa, a1;
  sqrt_rcp(g.gm1 * (ha - ka), aa, a1);
  const R la1 = ua - aa, la2 = ua + aa;
  const R lam0 = fabs(ua);
  R lam1 = fabs(la1), lam2 = fabs(la2);
  Flux5<R> o;
  o.lam = R(0);
  const bool near_fix = harten_near(l.u, r.u, l.a2, r.a2, ua, aa);
  if (want_lam || near_fix) {
    R al, ar;
    sqrt_fast(l.a2, al);
    sqrt_fast(r.a2, ar);
    if (near_fix) {
      const R le1 = R(0.05) * fmax(R(0), fmax(la1 - (l.u - al), (r.u - ar) - la1));
      const R le2 = R(0.05) * fmax(R(0), fmax(la2 - (l.u + al), (r.u + ar) - la2));
      if (!(lam1 > le1) && le1 > R(0)) lam1 = R(0.5) * (le1 + lam1 * lam1 / le1);
      if (!(lam2 > le2) && le2 > R(0)) lam2 = R(0.5) * (le2 + lam2 * lam2 / le2);
    }
    o.lam = max_pos(max_pos(fabs(l.u) + al, fabs(r.u) + ar), lam0 + aa);
  }
  const R ml = l.r * l.u, mr = r.r * r.u;
  const R d0 = mad(r.r, r.u, -ml), d2 = r.r - l.r;
  const R d3 = mad(r.r, r.h, -r.p) - mad(l.r, l.h, -l.p);
  const R dp = g.gm1 * mad(-ua, d0, mad(ka, d2, d3));
  const R cn = mad(-ua, d2, d0), da = dp * a1;
  const R w1 = (R(0.5) * lam1) * (cn - da), w2 = (R(0.5) * lam2) * (cn + da);
  const R z = mad(dp, a1 * a1, -d2);
  const R sm = w1 + w2, df = w2 - w1;
  const R drr = mad(-lam0, z, df * a1);
  const R e0 = mad(ua, drr, sm);
  o.f[0] = R(0.5) * (mad(ml, l.u, mad(mr, r.u, l.p + r.p)) - e0);
  o.f[1] = R(0);
  o.f[2] = R(0.5) * ((ml + mr) - drr);
  o.f[3] = R(0.5) * mad(-ka, drr, mad(-ua, sm, mad(-g.gamma1, df * aa, mad(ml, l.h, mr * r.h))));
  return o;
}

// per-lane constants of a tile: the records of the lane's left face, the offset over its right
// face, the cell's volume
template <class R> struct LineGeom {
  R dl, dr, idlr, wl, sl, wr, sr, dxl, dxr, ww, vol;
  int side;  // boundary of the left face: 0 or 1, else -1
};
template <class R> struct LinePhys {
  Gas<R> gas;
  int limiter;
  int bc[2];
};

template <class R>
__device__ __forceinline__ LineGeom<R> line_geom(const R* rec, const R* vol, int nc, bool per, int c) {
  LineGeom<R> g;
  // the face on the left of cell c, the one on its right; beyond the ends of a closed line the
  // faces repeat the end's, whose offset is 0
  const int f = per ? (c < 0 ? c + nc : (c > nc ? c - nc : c)) : min(max(c, 0), nc);
  const int fr = per ? (c + 1 < 0 ? c + 1 + nc : (c + 1 > nc ? c + 1 - nc : c + 1)) : min(max(c + 1, 0), nc);
  const int cc = per ? wrapi(c, nc) : min(max(c, 0), nc - 1);
  auto rd = [&](int fld, int k) -> R { return rec[size_t(fld) * (nc + 1) + k]; };
  g.dl = rd(F1_DL, f); g.dr = rd(F1_DR, f); g.idlr = rd(F1_IDLR, f);
  g.wl = rd(F1_WL, f); g.sl = rd(F1_SL, f); g.wr = rd(F1_WR, f); g.sr = rd(F1_SR, f);
  g.ww = rd(F1_WW, f);
  g.dxl = rd(F1_DX, f);
  g.dxr = rd(F1_DX, fr);
  g.vol = vol[cc];
  g.side = per ? -1 : (c == 0 ? 0 : (c == nc ? 1 : -1));
  return g;
}

// The reference state of an end and what the Riemann far field needs of it, once per launch
template <class R> struct LineRef {
  R q[3], n;            // {u, rho, p}; the normal into the domain
  R h, a2, ia2, rip;    // enthalpy, a^2 and its inverse, outgoing invariant u n + 2 a / (gamma - 1)
};
template <class R> __device__ __forceinline__ LineRef<R> line_ref(const LinePhys<R>& P, const R* const* gref, int side) {
  LineRef<R> f{};
  if (side < 0 || P.bc[side] == BC_WALL || P.bc[side] == BC_PERIODIC) return f;
#pragma unroll
  for (int v = 0; v < 3; ++v) f.q[v] = gref[side][v];
  f.n = side == 0 ? R(1) : R(-1);
  const St<R> s = st1(P.gas, f.q);
  f.h = s.h;
  f.a2 = s.a2;
  f.ia2 = rcp_fast(s.a2);
  R a;
  sqrt_fast(s.a2, a);
  f.rip = f.n * f.q[0] + R(2) * a * P.gas.gamma1;
  return f;
}
// Ghost state beyond an end of the line.  The Riemann far field is farfield_update's with the
// second velocity 0: the averaged velocity's direction is its sign, so the transverse test is
// a test of the sign.
template <class R> __device__ __forceinline__ void line_ghost(const LinePhys<R>& P, int bct, const LineRef<R>& f, const R* q, R* qg) {
  if (bct == BC_RIEMANN) {
    const Gas<R>& g = P.gas;
    const St<R> i = st1(g, q);
    const R ui = f.n * q[0], uf = f.n * f.q[0];
    R cr;
    sqrt_fast(f.q[1] * i.ir, cr);
    const R wl = rcp_fast(R(1) + cr), wr = R(1) - wl;
    const R ua = mad(wl, ui, wr * uf);
    R aa, ai;
    sqrt_fast(g.gm1 * (mad(wl, i.h, wr * f.h) - R(0.5) * (ua * ua)), aa);
    sqrt_fast(i.a2, ai);
    const bool in = ua > R(0);
    const R rim = mad(R(-2) * g.gamma1, ai, ui);
    const R ub = R(0.5) * (rim + f.rip);
    const R ab = (R(0.25) * g.gm1) * (f.rip - rim);
    const R ab2 = ab * ab;
    const R x = ab2 * (in ? f.ia2 : rcp_fast(i.a2));
    const R rb = (in ? f.q[1] : q[1]) * pow_gas(x, g.gamma1);
    const bool copy = ua < R(0) && !(g.fixes & FIX_FARFIELD_TRANSVERSE);
    const bool super = fabs(ua) > aa;
    const R b[3] = {f.n * ub, rb, rb * ab2 * g.inv_gamma};
#pragma unroll
    for (int v = 0; v < 3; ++v) qg[v] = copy ? q[v] : (super ? (in ? f.q[v] : q[v]) : b[v]);
  } else if (bct == BC_ENTROPY) {
    const R i4[4] = {q[0], R(0), q[1], q[2]}, f4[4] = {f.q[0], R(0), f.q[1], f.q[2]};
    R g4[4];
    farfield_update<R, BC_ENTROPY>(P.gas, f.n, R(0), i4, f4, g4);
    qg[0] = g4[0]; qg[1] = g4[2]; qg[2] = g4[3];
  } else {
#pragma unroll
    for (int v = 0; v < 3; ++v) qg[v] = f.q[v];
  }
}

// Residual of the tile's cells: q the lane's cell, qx the cell beyond it on lanes 0 and `last`
// (the lane of the right halo cell).  res and lam are valid on the lanes between.
// ghost: the ghost states of the two ends, computed meanwhile by another warp of the block (3
// values each; the block's barrier hands them over), or null: computed here from ref.
template <class R, int FK>
__device__ __forceinline__ void line_residual(const LinePhys<R>& P, const LineRef<R>& ref, const R* ghost, const LineGeom<R>& G,
                                              int lane, int last, const R* q, const R* qx, bool want_lam, R* res, R& lam) {
  constexpr unsigned all = 0xffffffffu;
  const int lim = P.limiter;
  R l[3], r[3], mi[3];
#pragma unroll
  for (int v = 0; v < 3; ++v) {
    R ql = __shfl_up_sync(all, q[v], 1);
    if (lane == 0) ql = qx[v];
    const R dq = q[v] - ql;
    R dqr = __shfl_down_sync(all, dq, 1);
    if (lane == last) dqr = qx[v] - q[v];
    const R m = mad(dqr, G.dxr, dq * G.dxl);  // gradient sum (spatial/lsqMetrics.h qmetrics, D2)
    const R ml = __shfl_up_sync(all, m, 1);
    mi[v] = G.side == 1 ? ml : m;
    if (lim != LIM_NOLIMIT1) {
      const R gc = dq * G.idlr;
      const R gl = mad(-dq, G.sl, ml * G.wl), gr = mad(-dq, G.sr, m * G.wr);
      l[v] = mad(G.dl, limit<R>(lim, gc, gl), ql);
      r[v] = mad(-G.dr, limit<R>(lim, gc, gr), q[v]);
    } else {
      l[v] = ql;
      r[v] = q[v];
    }
  }
  const int bct = G.side >= 0 ? P.bc[G.side] : BC_PERIODIC;
  if (ghost) __syncthreads();
  if (G.side >= 0 && bct != BC_WALL) {
    // the ghost state beyond the end; the lane's q is the interior cell's on either side (the
    // cells beyond a closed line repeat its last one)
    const bool int_right = G.side == 0;
    R qg[3];
    if (ghost) {
#pragma unroll
      for (int v = 0; v < 3; ++v) qg[v] = ghost[3 * G.side + v];
    } else {
      line_ghost(P, bct, ref, q, qg);
    }
#pragma unroll
    for (int v = 0; v < 3; ++v) {
      R qi = q[v];
      if (lim != LIM_NOLIMIT1) {
        const R dq = int_right ? (q[v] - qg[v]) : (qg[v] - q[v]);
        const R s = limit<R>(lim, dq * G.idlr, mi[v] * (int_right ? G.wr : G.wl));
        qi = int_right ? mad(-G.dl, s, q[v]) : mad(G.dl, s, q[v]);
      }
      l[v] = int_right ? qg[v] : qi;
      r[v] = int_right ? qi : qg[v];
    }
  }
  __syncwarp();
  Flux5<R> F;
  if constexpr (FK == FLUX_ROE || FK == FLUX_ROE_FACE) F = roe_flux_1d(P.gas, st1(P.gas, l), st1(P.gas, r), want_lam);
  else F = face_flux<R, FK>(P.gas, R(1), R(0), R(1), st1(P.gas, l), st1(P.gas, r), want_lam);
  if (bct == BC_WALL && G.side >= 0) {
    // the interior state moved to the face with the cell's gradient, normal into the domain;
    // res(interior) += F on both sides, stored as the face's (left - right) flux
    const bool int_right = G.side == 0;
    const R qw[4] = {mad(-mi[0], G.ww, q[0]), R(0), mad(-mi[1], G.ww, q[1]), mad(-mi[2], G.ww, q[2])};
    F = wall_flux(P.gas, int_right ? R(1) : R(-1), R(0), R(1), qw);
    if (!int_right) {
#pragma unroll
      for (int v = 0; v < 4; ++v) F.f[v] = -F.f[v];
    }
  }
  __syncwarp();
  const R f[3] = {F.f[0], F.f[2], F.f[3]};
#pragma unroll
  for (int v = 0; v < 3; ++v) res[v] = f[v] - __shfl_down_sync(all, f[v], 1);
  lam = F.lam + __shfl_down_sync(all, F.lam, 1);
}

// {rho u, rho, rho E} of {u, rho, p}, and back (spatial/eulerForwardUpdate.h:76-85)
template <class R> __device__ __forceinline__ void line_cons(const Gas<R>& g, const R* q, R* c) {
  c[0] = q[1] * q[0];
  c[1] = q[1];
  c[2] = mad(q[2], g.gamma1, q[1] * (R(0.5) * (q[0] * q[0])));
}
template <class R> __device__ __forceinline__ void line_prim(const Gas<R>& g, const R* c, R* q) {
  const R ir = rcp_near(c[1]);
  q[0] = c[0] * ir;
  q[1] = c[1];
  q[2] = g.gm1 * mad(-c[1], R(0.5) * (q[0] * q[0]), c[2]);
}
template <class R> __device__ __forceinline__ void update1(const Gas<R>& g, const R* q0, const R* tot, R fac, R* qn) {
  R c[3];
  line_cons(g, q0, c);
#pragma unroll
  for (int v = 0; v < 3; ++v) c[v] = mad(tot[v], fac, c[v]);
  line_prim(g, c, qn);
}

template <class R, int FK> __global__ void __launch_bounds__(32) stage1d_kernel(const Stage1DArgs<R> a) {
  const int nc = a.nc, lane = threadIdx.x, i0 = blockIdx.x * kLineCells;
  const bool per = a.bc[0] == BC_PERIODIC;
  const size_t n = size_t(nc);
  const int ncell = min(kLineCells, nc - i0), last = ncell + 1;
  const int c = i0 - 1 + min(lane, last);
  auto load = [&](int k, R* q) {
    const int cc = per ? wrapi(k, nc) : min(max(k, 0), nc - 1);
#pragma unroll
    for (int v = 0; v < 3; ++v) q[v] = a.q[v * n + cc];
  };
  R q[3], qx[3], res[3], lam;
  load(c, q);
  load(lane == 0 ? c - 1 : c + 1, qx);
  const LinePhys<R> P{a.gas, a.limiter, {a.bc[0], a.bc[1]}};
  const LineGeom<R> G = line_geom(a.rec, a.vol, nc, per, c);
  line_residual<R, FK>(P, line_ref(P, a.gref, G.side), nullptr, G, lane, last, q, qx, a.stage == 0, res, lam);
  const bool own = lane >= 1 && lane <= ncell;
  if (own && a.res_out) {
#pragma unroll
    for (int v = 0; v < 3; ++v) a.res_out[v * n + c] = res[v];
    if (a.stage == 0) a.res_out[3 * n + c] = lam;
  }
  if (a.mode == MODE_RES_MAXRATE || (a.mode == MODE_FUSED_LOCAL && a.norm_stage0 && a.stage == 0)) {
    R rate = own ? div_near(lam, G.vol) : R(0);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) rate = max_pos(rate, __shfl_xor_sync(0xffffffffu, rate, o));
    if (lane == 0) atomic_max_rate<R>(a.info, rate);
  }
  if (a.norm_stage0 && a.stage == 0) {
    R r2 = own ? res[1] * res[1] : R(0);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) r2 += __shfl_xor_sync(0xffffffffu, r2, o);
    if (lane == 0) atomicAdd(&a.info->resnorm2, double(r2));
  }
  if (a.mode == MODE_RES_MAXRATE || a.mode == MODE_RESIDUAL || !own) return;
  R tot[3] = {R(0), R(0), R(0)};
  for (int k = 0; k < a.stage; ++k)
#pragma unroll
    for (int v = 0; v < 3; ++v) tot[v] = mad(a.alpha[k], a.res_prev[k][v * n + c], tot[v]);
#pragma unroll
  for (int v = 0; v < 3; ++v) tot[v] = mad(a.alpha[a.stage], res[v], tot[v]);
  R fac;
  if (a.mode == MODE_FUSED_GLOBAL) {
    fac = div_near(a.beta * R(a.info->dt), G.vol);
  } else {
    const R l0 = (a.stage == 0) ? lam : a.res_prev[0][3 * n + c];
    fac = div_near(a.beta * a.cfl, l0);
  }
  R q0[3], qn[3];
#pragma unroll
  for (int v = 0; v < 3; ++v) q0[v] = a.q0[v * n + c];
  update1(a.gas, q0, tot, fac, qn);
#pragma unroll
  for (int v = 0; v < 3; ++v) a.q_out[v * n + c] = qn[v];
  const R chk[4] = {qn[0], R(0), qn[1], qn[2]};
  flag_nonphysical(a.info, chk, c);
}

// ---- a short line's steps in one launch
// Lines of up to 960 cells take their steps in one cluster of up to eight blocks, a warp per
// tile: the state, the step's start and the stage residuals stay in registers, neighbouring
// tiles exchange two cells a side through distributed shared memory, and the global timestep
// is a maximum over the cluster -- five cluster barriers per ssp34 step instead of six
// launches and their trips through L2.  Where an end has a far field, a warp more in its block
// computes the ghost state while the tile's warp reconstructs.  What bounds it: one warp's FP64
// instructions, about 190 a stage at 64 cycles each.  Sod's tube, 128 cells, Roe + MC, ssp34,
// FP64: 146 us per step at first (256-cell tiles on one SM, six launches), 64 with the ghost
// state in the tile's warp, 39 now.
constexpr int kLineBlocks = 8, kLineWarps = 4, kLineChunk = 64;  // steps of one launch
constexpr int kLineMax = kLineBlocks * kLineWarps * kLineCells;
template <class R> struct LineRunArgs {
  int nc, nsteps, tiles, warps;  // tiles of the line, warps per block
  LinePhys<R> P;
  const R* rec;
  const R* vol;
  const R* gref[2];
  R* q;
  int nst, global;
  R alpha[4][4], beta[4];
  R cfl;
  double dcfl;
  StepInfo* info;
};
template <class R> struct LineMail {
  R cell[2][2][2][3];  // by parity of the exchange, side (0: from the left), distance, variable
};
// dynamic shared memory that leaves room for one block per SM: two on one SM would share its
// FP64 pipe
constexpr int kLineSmem = 120 * 1024;

// (its aligned form takes the warp's lanes together, whatever branches came before)
__device__ __forceinline__ void cluster_barrier() {
  __syncwarp();
  asm volatile("barrier.cluster.arrive.release.aligned;\nbarrier.cluster.wait.acquire.aligned;\n" ::: "memory");
}
template <class T> __device__ __forceinline__ T* cluster_ptr(T* p, unsigned block) {
  uint64_t out;
  asm("mapa.u64 %0, %1, %2;\n" : "=l"(out) : "l"(reinterpret_cast<uint64_t>(p)), "r"(block));
  return reinterpret_cast<T*>(out);
}
// maximum over the warp of bit patterns of non-negative values
__device__ __forceinline__ unsigned long long warp_max_bits(unsigned long long b) {
  const unsigned hi = __reduce_max_sync(0xffffffffu, unsigned(b >> 32));
  const unsigned lo = __reduce_max_sync(0xffffffffu, unsigned(b >> 32) == hi ? unsigned(b) : 0u);
  return (unsigned long long)hi << 32 | lo;
}

// x / d by d's inverse r, taken once per launch: the product corrected by its remainder, in three
// FP64 instructions the quotient rounded once (P. W. Markstein, "Computation of elementary functions
// on the IBM RISC System/6000 processor", 1990), where the product alone is off by an ulp.  FP32
// divides, as the launches per stage do.
__device__ __forceinline__ float line_div(float x, float d, float) { return div_near(x, d); }
__device__ __forceinline__ double line_div(double x, double d, double r) {
  const double q = x * r;
  // (an infinite or NaN quotient stays)
  if ((f64_bits(q) & 0x7fffffffffffffffLL) >= 0x7ff0000000000000LL) return q;
  return fma(fma(-q, d, x), r, q);
}

template <class R, int FK>
__global__ void __launch_bounds__(32 * (kLineWarps + 1)) line_run_kernel(const __grid_constant__ LineRunArgs<R> a) {
  __shared__ LineMail<R> mail[kLineWarps];
  __shared__ R end_q[2][3], end_ghost[2][3];  // the ends' cells and ghost states
  __shared__ unsigned long long rates[2][kLineBlocks * kLineWarps];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int nt = a.tiles;
  const bool per = a.P.bc[0] == BC_PERIODIC;
  const bool ext = blockDim.x > unsigned(32 * a.warps);  // the block has a ghost warp
  if (warp == a.warps) {
    // the ghost warp: lane 0 the low end, lane 1 the high end, where this block has them
    const int side = (lane == 0 && blockIdx.x == 0) ? 0 : ((lane == 1 && blockIdx.x == gridDim.x - 1) ? 1 : -1);
    const int bct = side >= 0 ? a.P.bc[side] : BC_WALL;
    const LineRef<R> f = line_ref(a.P, a.gref, side);
    cluster_barrier();
#pragma unroll 1
    for (int step = 0; step < a.nsteps; ++step)
#pragma unroll 1
      for (int s = 0; s < a.nst; ++s) {
        if (side >= 0 && bct != BC_WALL) {
          R q[3], g[3];
#pragma unroll
          for (int v = 0; v < 3; ++v) q[v] = end_q[side][v];
          line_ghost(a.P, bct, f, q, g);
#pragma unroll
          for (int v = 0; v < 3; ++v) end_ghost[side][v] = g[v];
        }
        __syncwarp();
        __syncthreads();
        if (s == 0 && a.global) cluster_barrier();
        cluster_barrier();
      }
    cluster_barrier();
    return;
  }
  const int tile = int(blockIdx.x) * a.warps + warp;
  const bool live = tile < nt;
  const int nc = a.nc;
  const size_t n = size_t(nc);
  // the cells divided evenly over the tiles
  const int i0 = live ? int((long long)nc * tile / nt) : 0, i1 = live ? int((long long)nc * (tile + 1) / nt) : 1;
  const int ncell = i1 - i0, last = ncell + 1;
  const int c = i0 - 1 + min(lane, last);
  const bool own = live && lane >= 1 && lane <= ncell;
  const LineGeom<R> G = line_geom(a.rec, a.vol, nc, per, c);
  const R ivol = div_near(R(1), G.vol);
  R q[3], qx[3];
  auto load = [&](int k, R* x) {
    const int cc = per ? wrapi(k, nc) : min(max(k, 0), nc - 1);
#pragma unroll
    for (int v = 0; v < 3; ++v) x[v] = a.q[v * n + cc];
  };
  load(c, q);
  load(lane == 0 ? c - 1 : c + 1, qx);
  // the mailboxes this lane writes: its cell is the left or right neighbour tile's halo
  const int tl = tile > 0 ? tile - 1 : (per ? nt - 1 : -1), tr = tile + 1 < nt ? tile + 1 : (per ? 0 : -1);
  R* to_left = nullptr;
  R* to_right = nullptr;
  if (own && tl >= 0 && lane <= 2) to_left = cluster_ptr(&mail[tl % a.warps].cell[0][1][lane - 1][0], unsigned(tl / a.warps));
  if (own && tr >= 0 && lane >= ncell - 1)
    to_right = cluster_ptr(&mail[tr % a.warps].cell[0][0][ncell - lane][0], unsigned(tr / a.warps));
  constexpr int parity_stride = 12;  // values of one parity in LineMail
  const LineRef<R> ref{};
  const R* ghost = ext ? &end_ghost[0][0] : nullptr;
  // the interior cell of an end, for the ghost warp
  const int end = per || !own ? -1 : (c == 0 ? 0 : (c == nc - 1 ? 1 : -1));
  if (end >= 0) {
#pragma unroll
    for (int v = 0; v < 3; ++v) end_q[end][v] = q[v];
  }
  unsigned exchange = 0;
  double t = 0.0, dt_last = 0.0;
  if (tile == 0 && lane == 0) t = a.info->t;
  cluster_barrier();  // every block of the cluster runs before its shared memory is written
#pragma unroll 1
  for (int step = 0; step < a.nsteps; ++step) {
    const bool final_step = step == a.nsteps - 1;
    // the earlier stages' residuals as their sum: each row of every table weighs them alike
    // (ode.h:107-197)
    R c0[3], rs[3] = {R(0), R(0), R(0)}, fac0 = R(0), lam0 = R(1);
    line_cons(a.P.gas, q, c0);
#pragma unroll 1
    for (int s = 0; s < a.nst; ++s) {
      R res[3], lam;
      line_residual<R, FK>(a.P, ref, ghost, G, lane, last, q, qx, s == 0, res, lam);
      if (s == 0) {
        const R rate = own ? line_div(lam, G.vol, ivol) : R(0);
        // a NaN or negative rate does not count, as in atomic_max_rate
        const unsigned long long bits =
            rate > R(0) ? (unsigned long long)__double_as_longlong(double(rate)) : 0ull;
        unsigned long long top = warp_max_bits(bits);
        if (a.global) {
          unsigned long long* slot = &rates[step & 1][tile];
          if (lane < int(gridDim.x) && live) *cluster_ptr(slot, unsigned(lane)) = top;
          cluster_barrier();
          top = warp_max_bits(lane < nt ? rates[step & 1][lane] : 0ull);
          const double r = fmax(DBL_MIN, __longlong_as_double((long long)top));
          const R dt = R(a.dcfl / r);
          dt_last = double(dt);
          t += dt_last;
          fac0 = dt;
          if (final_step && tile == 0 && lane == 0) a.info->maxrate = top;
        } else {
          fac0 = a.cfl;
          lam0 = lam;
          if (final_step && lane == 0 && live) atomicMax(&a.info->maxrate, top);
        }
        if (final_step) {
          R r2 = own ? res[1] * res[1] : R(0);
#pragma unroll
          for (int o = 16; o > 0; o >>= 1) r2 += __shfl_xor_sync(0xffffffffu, r2, o);
          if (lane == 0 && live) atomicAdd(&a.info->resnorm2, double(r2));
        }
      }
      // rungeKuttaAccumulation (timestepping/rungeKutta.h:172-197) and the update
      R cn[3];
      const R fac = a.global ? line_div(a.beta[s] * fac0, G.vol, ivol)
                             : line_div(a.beta[s] * fac0, lam0, rcp_fast(lam0));
#pragma unroll
      for (int v = 0; v < 3; ++v) {
        const R tot = mad(a.alpha[s][s], res[v], s > 0 ? a.alpha[s][0] * rs[v] : R(0));
        cn[v] = mad(tot, fac, c0[v]);
        rs[v] = rs[v] + res[v];
      }
      R qn[3];
      line_prim(a.P.gas, cn, qn);
      if (own) {
        const R chk[4] = {qn[0], R(0), qn[1], qn[2]};
        flag_nonphysical(a.info, chk, c);
      }
      // the halo cells from the neighbouring tiles; those beyond a closed end repeat the last cell
      const unsigned p = exchange++ & 1u;
#pragma unroll
      for (int v = 0; v < 3; ++v) {
        if (to_left) to_left[p * parity_stride + v] = qn[v];
        if (to_right) to_right[p * parity_stride + v] = qn[v];
        if (end >= 0) end_q[end][v] = qn[v];
      }
      cluster_barrier();
      const LineMail<R>& mb = mail[warp];
#pragma unroll
      for (int v = 0; v < 3; ++v) {
        const R first = __shfl_down_sync(0xffffffffu, qn[v], 1), final = __shfl_up_sync(0xffffffffu, qn[v], 1);
        if (lane == 0) {
          q[v] = tl >= 0 ? mb.cell[p][0][0][v] : first;
          qx[v] = tl >= 0 ? mb.cell[p][0][1][v] : first;
        } else if (lane >= last) {
          q[v] = tr >= 0 ? mb.cell[p][1][0][v] : final;
          qx[v] = tr >= 0 ? mb.cell[p][1][1][v] : final;
        } else {
          q[v] = qn[v];
        }
      }
    }
  }
  if (own) {
#pragma unroll
    for (int v = 0; v < 3; ++v) a.q[v * n + c] = q[v];
  }
  if (tile == 0 && lane == 0 && a.global) {
    a.info->dt = dt_last;
    a.info->t = t;
  }
  cluster_barrier();  // no block leaves while another may still write to its shared memory
}

// the run's shared memory, allowed on the device of the calling thread
template <class R, int FK> cudaError_t prepare_run() {
  return cudaFuncSetAttribute(line_run_kernel<R, FK>, cudaFuncAttributeMaxDynamicSharedMemorySize, kLineSmem);
}
// the cluster of a short line: as many blocks as tiles up to eight, then more warps a block
template <class R, int FK> cudaError_t go_run(const LineRunArgs<R>& args, cudaStream_t s) {
  LineRunArgs<R> a = args;
  a.tiles = (a.nc + kLineCells - 1) / kLineCells;
  a.warps = (a.tiles + kLineBlocks - 1) / kLineBlocks;
  const int blocks = (a.tiles + a.warps - 1) / a.warps;
  // a warp more for the ghost states, unless neither end has one to compute
  auto plain = [](int bc) { return bc == BC_PERIODIC || bc == BC_WALL; };
  const int ghost = plain(a.P.bc[0]) && plain(a.P.bc[1]) ? 0 : 1;
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(unsigned(blocks));
  cfg.blockDim = dim3(unsigned(32 * (a.warps + ghost)));
  cfg.dynamicSmemBytes = kLineSmem;
  cfg.stream = s;
  cudaLaunchAttribute attr{};
  attr.id = cudaLaunchAttributeClusterDimension;
  attr.val.clusterDim.x = unsigned(blocks);
  attr.val.clusterDim.y = attr.val.clusterDim.z = 1;
  cfg.attrs = &attr;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, line_run_kernel<R, FK>, a);
}
template <class R> cudaError_t launch_line_run(const LineRunArgs<R>& a, int flux, cudaStream_t s);
// the kernel of a flux made ready on the current device (at every mesh upload: a process may use
// several devices)
template <class R> cudaError_t prepare_line_run(int flux);

// stage-0 update of the 1D path with the global timestep
template <class R>
__global__ void update0_1d_kernel(int nc, Gas<R> g, const R* __restrict__ q0, const R* __restrict__ res0,
                                  const R* __restrict__ vol, R alpha00, R beta0, double cfl, StepInfo* info,
                                  R* __restrict__ q_out) {
  const R dt = global_dt<R>(info, cfl);
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    info->dt = double(dt);
    info->t += double(dt);
  }
  const size_t n = size_t(nc);
  for (size_t c = blockIdx.x * size_t(blockDim.x) + threadIdx.x; c < n; c += size_t(gridDim.x) * blockDim.x) {
    R tot[3], q[3], qn[3];
#pragma unroll
    for (int v = 0; v < 3; ++v) { tot[v] = R(0) + alpha00 * res0[v * n + c]; q[v] = q0[v * n + c]; }
    update1(g, q, tot, div_near(beta0 * dt, vol[c]), qn);
#pragma unroll
    for (int v = 0; v < 3; ++v) q_out[v * n + c] = qn[v];
    const R chk[4] = {qn[0], R(0), qn[1], qn[2]};
    flag_nonphysical(info, chk, int(c));
  }
}

// Stage update of the 1D path from stored stage residuals (the update of the fused
// stage kernel as a kernel of its own, for residuals changed between the two: residual
// smoothing).  res[k] holds 4 planes (3 flux sums and lambda) of stage k; global dt: at
// stage 0 from the recorded max rate (and stored), later stages read it; local dt: the
// stage-0 lambda.
template <class R> struct Update1DArgs {
  int nc;
  Gas<R> gas;
  const R* q0;
  const R* res[4];
  R alpha[4];
  int stage;
  R beta;
  int global;
  double cfl;
  StepInfo* info;
  const R* vol;
  R* q_out;
};
template <class R> __global__ void update_stage_1d_kernel(const Update1DArgs<R> u) {
  const size_t n = size_t(u.nc);
  R dt = R(0);
  if (u.global) {
    if (u.stage == 0) {
      dt = global_dt<R>(u.info, u.cfl);
      if (blockIdx.x == 0 && threadIdx.x == 0) {
        u.info->dt = double(dt);
        u.info->t += double(dt);
      }
    } else {
      dt = R(u.info->dt);
    }
  }
  for (size_t c = blockIdx.x * size_t(blockDim.x) + threadIdx.x; c < n; c += size_t(gridDim.x) * blockDim.x) {
    R tot[3] = {R(0), R(0), R(0)};
    for (int k = 0; k <= u.stage; ++k)
#pragma unroll
      for (int v = 0; v < 3; ++v) tot[v] += u.alpha[k] * u.res[k][v * n + c];
    const R fac = u.global ? (u.beta * dt) / u.vol[c] : (u.beta * R(u.cfl)) / u.res[0][3 * n + c];
    R q[3], qn[3];
#pragma unroll
    for (int v = 0; v < 3; ++v) q[v] = u.q0[v * n + c];
    update1(u.gas, q, tot, fac, qn);
#pragma unroll
    for (int v = 0; v < 3; ++v) u.q_out[v * n + c] = qn[v];
    const R chk[4] = {qn[0], R(0), qn[1], qn[2]};
    flag_nonphysical(u.info, chk, int(c));
  }
}

template <class R> cudaError_t launch_stage1d(const Stage1DArgs<R>& a, int flux, cudaStream_t s);

}  // namespace hc
