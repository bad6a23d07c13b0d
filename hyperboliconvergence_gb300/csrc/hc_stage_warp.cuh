// hc_stage_warp.cuh -- the FP32 stage kernel of the 2D Euler path (primitive basis, the common
// limiters): one warp advances a strip of 28 columns over a run of rows, without shared tiles
// or block barriers.
//
// A lane is one column of the strip (28 cells and two halo columns either side).  Marching down
// the rows it keeps in registers the states of three rows, the gradient sums of two and the
// flux through the row's upper face, so every row's state is loaded once and every i-face is
// evaluated once (the first row of a run repeats one face and two gradient rows); what a j-face
// needs of the neighbouring column comes by warp shuffles: the jump to it, the state
// reconstructed on its side of the face, and the next face's flux.
//
// The face records come from a copy of the geometry laid out for this kernel (pack_strips):
// for each strip and row the 27 values x 32 lanes of one row's work are 3,456 contiguous bytes,
// padded per strip, so one cp.async.bulk per row lands them in the warp's three-slot ring in
// shared memory while the two rows before it are computed, whatever the mesh's width.  The
// waits are bounded (a copy that never lands marks the step ST_TIMEOUT).  The records hold the
// limiter's arguments scaled by the distance between the cell centres, w (dl + dr),
// s (dl + dr), dl/(dl + dr) and dr/(dl + dr): the limiters are homogeneous, and the division
// by that distance disappears.
//
// What bounds it: instruction issue (59% of the issue slots at four warps per scheduler, no pipe
// above 30%; 1,190 thread instructions per cell and stage, halo lanes and lead-in rows
// included).  The tiled kernel before it (8 x 32 cells, halo and gradient tiles in shared
// memory, four block barriers) issued 1,577 at 45%, waiting on barriers and on the j-face
// records.  512 x 1024 O-grid, Roe + van Albada: 0.168 -> 0.115 ms per ssp34 step; a batch of 24
// uneven quadrant problems, SLAU, 20 steps, uploads and downloads included: 18.8 -> 15.8 ms.
// Four blocks of four warps per SM: 126 registers hold a pass without spills (with the edge
// faces' code out of line the calls cost 48 bytes of spills and 15% of the time), and 512 x 1024
// in runs of 8 rows is one wave of 2,368 warps.
//
// The stage residuals of the alpha/beta tables are kept as their running sum (each row of every
// table weighs the earlier stages alike, ode.h:107-197), so a later stage reads and writes one
// 4-plane buffer whatever its number.
#pragma once

#include "hc_kernels.cuh"

#include <algorithm>
#include <cmath>

namespace hc {

constexpr int kStripCells = 28;                      // columns a strip owns
constexpr int kStripRowsBefore = 3;                  // record rows before row 0 (the run's lead-in)
// fields of a record row r, in the order of the first and last rows' needs: the gradient sums of
// row r + 1 (left j-face and lower i-face offsets), the i-face r + 1, the volume of row r, the
// j-face on the left of row r + 1
enum StripField { S_DXJ = 0, S_DXI = 2, S_IF = 4, S_VOL = 15, S_JF = 16, S_FIELDS = 27 };
// fields of a face within S_IF / S_JF
enum StripFace { P_NX = 0, P_NY, P_A, P_CL, P_CR, P_WLX, P_WLY, P_SL, P_WRX, P_WRY, P_SR, P_FIELDS };
constexpr int kStripRow = S_FIELDS * 32;             // floats of one strip and row
constexpr int kStripSlots = 3;
constexpr int kStripWarps = 4;                       // warps of a block
constexpr size_t kStripSmem = size_t(kStripWarps) * kStripSlots * (kStripRow * sizeof(float) + sizeof(uint64_t));

__host__ __device__ inline int strip_count(int nj) { return (nj + kStripCells - 1) / kStripCells; }
// floats of a mesh's packed records
__host__ __device__ inline size_t strip_floats(int ni, int nj) {
  return size_t(strip_count(nj)) * (ni + kStripRowsBefore) * kStripRow;
}

// Rows of a run, at most, for the given meshes (a mesh's rows are divided evenly over
// ceil(ni / rows) runs): a launch takes the waves its runs make of the 152 SMs' resident warps,
// times a run's rows and its lead-in (1.7 rows' work).  Small meshes are cut finer, so that
// every SM has work, and large ones so that the last wave is full.  Measured, ms per step: 512 x
// 1024 with 8 rows (one wave) 0.115, with 16 (half a wave: each warp's latency is exposed) 0.24;
// a batch of 24 meshes, 2.27 M cells, with 8 rows (4.2 waves) 0.64, by this rule (2 waves) 0.57;
// 96 small ones, 0.47 M cells, 0.255 and 0.20.
inline int strip_runs(int ni, int rows) { return (ni + rows - 1) / rows; }
template <class NI, class NJ> inline int strip_run_rows(int n, NI ni, NJ nj, int sms) {
  constexpr int kResident = 16;  // warps per SM
  int best = 1;
  double cost = 1e300;
  for (int rows = 1; rows <= 64; ++rows) {
    long long items = 0;
    int longest = 0;
    bool fits = true;  // a work item is packed in 16 bits within its instance
    for (int k = 0; k < n; ++k) {
      const int runs = strip_runs(ni(k), rows);
      const long long m = (long long)strip_count(nj(k)) * runs;
      items += m;
      longest = std::max(longest, (ni(k) + runs - 1) / runs);
      fits = fits && (n == 1 || m <= 0xffff);
    }
    const double c = std::ceil(double(items) / (double(sms) * kResident)) * (longest + 1.7);
    if (fits && c < cost) { cost = c; best = rows; }
  }
  return best;
}

// Pack the FP64 face records (FREC planes of the i- and j-faces) and volumes of a mesh
// (hc_strip_pack.cu): rows and columns outside the mesh wrap on periodic sides; elsewhere they
// take the nearest face with zero offsets, so that they add nothing.
cudaError_t pack_strips(const double* fi, const double* fj, const double* vol, int ni, int nj, const int bc[4],
                        float* out, cudaStream_t s);

struct StripArgs {
  StageArgs<float> a;
  int strips, runs;  // strips of the mesh, runs of rows
};

// ---- limiters on arguments scaled by the centres' distance
template <int LIM> __device__ __forceinline__ float strip_limit(float a, float b) {
  if constexpr (LIM == LIM_VANALBADA) {
    const float ab = a * b;
    const float s = (ab * (a + b)) * rcp_f32(fmaf(a, a, fmaf(b, b, FLT_MIN)));
    return ab <= 0.f ? 0.f : s;
  } else if constexpr (LIM == LIM_VANLEER) {
    const float ab = a * b;
    const float s = (ab + ab) * rcp_f32(a + b);
    return ab <= 0.f ? 0.f : s;
  } else {
    return limit<float>(LIM, a, b);
  }
}

// Flux through a non-periodic boundary face: wall, or a ghost state on the far side (fixed,
// Riemann or entropy).  s holds the interior cell's state and gradient sums and the face's
// weights.  (Out of line it costs spills around the call: the main loop fills the registers.)
struct StripEdge {
  float q[4], m[8];
  float nx, ny, A;
  float wx, wy;    // one-sided gradient weights, scaled
  float wwx, wwy;  // wall extrapolation weights
};
template <int FK, int LIM>
__device__ __forceinline__ void strip_edge_flux(const StageArgs<float>& a, int side, int kf, const StripEdge& s,
                                             bool want_lam, Flux5<float>& F) {
  const bool int_right = side == 0 || side == 2;
  const int bct = a.bc[side];
  if (bct == BC_WALL) {
    float qw[4];
#pragma unroll
    for (int v = 0; v < 4; ++v) qw[v] = s.q[v] - fmaf(s.m[2 * v + 1], s.wwy, s.m[2 * v] * s.wwx);
    F = wall_flux(a.gas, s.nx, s.ny, s.A, qw, false);
    return;
  }
  const int nfs = side < 2 ? a.nj : a.ni;
  float qf[4], qg[4];
#pragma unroll
  for (int v = 0; v < 4; ++v) qf[v] = a.gref[side][size_t(v) * nfs + kf];
  const float sgn = int_right ? 1.f : -1.f;  // normal into the domain
  if (bct == BC_RIEMANN) farfield_update<float, BC_RIEMANN>(a.gas, sgn * s.nx, sgn * s.ny, s.q, qf, qg, false, nullptr);
  else if (bct == BC_ENTROPY)
    farfield_update<float, BC_ENTROPY>(a.gas, sgn * s.nx, sgn * s.ny, s.q, qf, qg, false, nullptr);
  else {
#pragma unroll
    for (int v = 0; v < 4; ++v) qg[v] = qf[v];
  }
  float qi[4];
#pragma unroll
  for (int v = 0; v < 4; ++v) {
    const float dq = int_right ? (s.q[v] - qg[v]) : (qg[v] - s.q[v]);
    const float sl = strip_limit<LIM>(dq, fmaf(s.m[2 * v + 1], s.wy, s.m[2 * v] * s.wx));
    qi[v] = fmaf(int_right ? -0.5f : 0.5f, sl, s.q[v]);
  }
  St<float> l, r;
  basis_state2(a.gas, int_right ? qg : qi, int_right ? qi : qg, false, l, r);
  F = face_flux<float, FK>(a.gas, s.nx, s.ny, s.A, l, r, want_lam);
}

// the ring of record rows of one warp
struct StripRing {
  float* slot;       // kStripSlots x kStripRow floats
  uint64_t* bar;     // kStripSlots barriers
  unsigned used;     // rows fetched so far: slot and phase of the next fetch
  unsigned read;     // rows waited for so far
  bool staged, dead;
};

// fetch the first n floats of a record row into the ring's next slot (every lane; the warp has
// finished reading that slot)
__device__ __forceinline__ void strip_fetch(StripRing& ring, const float* src, int n, int lane, bool stall) {
  if (ring.dead) return;
  const unsigned k = ring.used % kStripSlots;
  ring.used += 1;
  float* dst = ring.slot + k * kStripRow;
  if (ring.staged) {
    if (lane == 0) {
      mbar_expect_tx(&ring.bar[k], unsigned(n) * 4u + (stall ? 16u : 0u));
      asm volatile(
          "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];\n" ::"r"(
              smem_u32(dst)),
          "l"(reinterpret_cast<uint64_t>(src)), "r"(unsigned(n) * 4u), "r"(smem_u32(&ring.bar[k]))
          : "memory");
    }
  } else {
    for (int i = 4 * lane; i < n; i += 128)
      *reinterpret_cast<float4*>(dst + i) = *reinterpret_cast<const float4*>(src + i);
  }
}
__device__ __forceinline__ bool strip_poll(uint64_t* bar, unsigned parity) {
  unsigned ok;
  asm volatile(
      "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}\n"
      : "=r"(ok)
      : "r"(smem_u32(bar)), "r"(parity)
      : "memory");
  return ok != 0;
}
// wait for the next fetched row (at most kCopyWaitNs) and return its slot
__device__ __forceinline__ const float* strip_wait(StripRing& ring, StepInfo* info) {
  const unsigned k = ring.read % kStripSlots, parity = (ring.read / kStripSlots) & 1u;
  ring.read += 1;
  if (ring.staged && !ring.dead && !strip_poll(&ring.bar[k], parity)) {
    const unsigned long long t0 = globaltimer_ns();
    bool late = false;
    while (!late && !strip_poll(&ring.bar[k], parity)) late = globaltimer_ns() - t0 > kCopyWaitNs;
    if (__any_sync(0xffffffffu, late)) {
      ring.dead = true;  // no further copies or waits; the rows computed from here are discarded with the step
      atomicCAS(&info->status, ST_OK, ST_TIMEOUT);
    }
  }
  __syncwarp();
  return ring.slot + k * kStripRow;
}

// One run of rows [r0, r1) of strip w.
template <int FK, int LIM>
__device__ __forceinline__ void strip_run(const StageArgs<float>& a, const float* pk, int w, int r0, int r1,
                                          StripRing& ring) {
  const int lane = threadIdx.x & 31;
  const int ni = a.ni, nj = a.nj;
  const size_t ncell = size_t(ni) * nj;
  const bool per_i = a.bc[0] == BC_PERIODIC, per_j = a.bc[2] == BC_PERIODIC;
  const int c = w * kStripCells - 2 + lane;  // this lane's column
  const int cq = per_j ? wrapi(c, nj) : min(max(c, 0), nj - 1);
  const bool own = lane >= 2 && lane < 30 && c < nj;
  // the lane's left face lies on a boundary: 2 or 3, else -1
  const int jside = per_j ? -1 : (c == 0 ? 2 : (c == nj ? 3 : -1));
  const bool edge_j = __any_sync(0xffffffffu, jside >= 0 && lane >= 2 && lane <= 30);
  const bool want_lam = a.stage == 0;
  const Gas<float>& g = a.gas;
  const float* rows = pk + size_t(w) * (ni + kStripRowsBefore) * kStripRow;  // record row r at (r + 3) kStripRow
  auto recrow = [&](int r) { return rows + size_t(r + kStripRowsBefore) * kStripRow; };
  // the lane's cell in row r (fewer than 2^28 cells: 32-bit offsets from the planes' bases)
  auto qcell = [&](int r) -> unsigned {
    int rr = r;
    if (per_i) { if (rr < 0 || rr >= ni) rr = wrapi(rr, ni); }
    else rr = min(max(rr, 0), ni - 1);
    return unsigned(rr) * unsigned(nj) + unsigned(cq);
  };

  // The march: pass r (from r0 - 1) forms the gradient sums of row r + 1, the j-faces of row
  // r + 1 and the i-face between rows r and r + 1, and completes row r.  Its record row is r;
  // record row r0 - 2 serves the gradient sums of row r0 - 1 before the first pass.
  auto fetch_row = [&](int r, bool stall) {
    strip_fetch(ring, recrow(r), (r == r1 - 1 ? S_JF : S_FIELDS) * 32, lane, stall);
  };
  strip_fetch(ring, recrow(r0 - 2), S_IF * 32, lane, false);
  fetch_row(r0 - 1, false);
  fetch_row(r0, a.stall_copy != 0);

  // the records do not depend on the stage before: their copies are under way while it ends
  chain_wait<true>();
  float qa[4], qb[4], qc[4], qn[4];  // rows r, r + 1, r + 2, r + 3
  {
    const unsigned k0 = qcell(r0 - 2), k1 = qcell(r0 - 1), k2 = qcell(r0), k3 = qcell(r0 + 1);
#pragma unroll
    for (int v = 0; v < 4; ++v) {
      const float* p = a.q + v * ncell;
      qa[v] = p[k0];
      qb[v] = p[k1];
      qc[v] = p[k2];
      qn[v] = p[k3];
    }
  }
  // offset of the i-face between rows r and r + 1
  float dxi, dyi;
  {
    const float* p = recrow(r0 - 3) + S_DXI * 32 + lane;
    dxi = p[0];
    dyi = p[32];
  }
  float ma[8], mb[8];   // gradient sums of rows r, r + 1
  float dl[4], dr[4];   // jumps over the left and right faces in row r + 1
  float fi[4], fil = 0.f;  // flux through the i-face r (the upper face of row r)
  float fj[4], fjl = 0.f;  // net j-flux of row r
#pragma unroll
  for (int v = 0; v < 4; ++v) { fi[v] = fj[v] = 0.f; ma[2 * v] = ma[2 * v + 1] = 0.f; }

  // gradient sums (lsq/qmetric.ipp) of row r + 1 from rows r, r + 1, r + 2
  auto gradient = [&](const float* s) {
    const float xj0 = s[S_DXJ * 32 + lane], yj0 = s[(S_DXJ + 1) * 32 + lane];
    const float xj1 = s[S_DXJ * 32 + lane + 1], yj1 = s[(S_DXJ + 1) * 32 + lane + 1];
    const float xi1 = s[S_DXI * 32 + lane], yi1 = s[(S_DXI + 1) * 32 + lane];
#pragma unroll
    for (int v = 0; v < 4; ++v) {
      const float left = __shfl_up_sync(0xffffffffu, qb[v], 1);
      dl[v] = qb[v] - left;
      dr[v] = __shfl_down_sync(0xffffffffu, dl[v], 1);
      const float a0 = qb[v] - qa[v], a1 = qc[v] - qb[v];
      mb[2 * v] = fmaf(dr[v], xj1, fmaf(dl[v], xj0, fmaf(a1, xi1, a0 * dxi)));
      mb[2 * v + 1] = fmaf(dr[v], yj1, fmaf(dl[v], yj0, fmaf(a1, yi1, a0 * dyi)));
    }
    dxi = xi1;
    dyi = yi1;
  };
  // flux through the i-face r + 1, between rows r and r + 1
  auto iface = [&](const float* s, int r, Flux5<float>& F) {
    const float* f = s + S_IF * 32 + lane;
    const int face = r + 1;
    if (!per_i && (face == 0 || face == ni)) {
      const bool lo = face == 0;
      StripEdge e;
#pragma unroll
      for (int v = 0; v < 4; ++v) e.q[v] = lo ? qb[v] : qa[v];
#pragma unroll
      for (int v = 0; v < 8; ++v) e.m[v] = lo ? mb[v] : ma[v];
      e.nx = f[P_NX * 32]; e.ny = f[P_NY * 32]; e.A = f[P_A * 32];
      e.wx = f[(lo ? P_WRX : P_WLX) * 32]; e.wy = f[(lo ? P_WRY : P_WLY) * 32];
      e.wwx = f[(lo ? P_WLX : P_WRX) * 32]; e.wwy = f[(lo ? P_WLY : P_WRY) * 32];
      strip_edge_flux<FK, LIM>(a, lo ? 0 : 1, cq, e, want_lam, F);
      return;
    }
    float ql[4], qr[4];
    {
      const float cl = f[P_CL * 32], cr = f[P_CR * 32];
      const float wlx = f[P_WLX * 32], wly = f[P_WLY * 32], sl = f[P_SL * 32];
      const float wrx = f[P_WRX * 32], wry = f[P_WRY * 32], sr = f[P_SR * 32];
#pragma unroll
      for (int v = 0; v < 4; ++v) {
        const float dq = qb[v] - qa[v];
        const float gl = fmaf(-dq, sl, fmaf(ma[2 * v + 1], wly, ma[2 * v] * wlx));
        const float gr = fmaf(-dq, sr, fmaf(mb[2 * v + 1], wry, mb[2 * v] * wrx));
        ql[v] = fmaf(cl, strip_limit<LIM>(dq, gl), qa[v]);
        qr[v] = fmaf(-cr, strip_limit<LIM>(dq, gr), qb[v]);
      }
    }
    St<float> l, rr;
    basis_state2(g, ql, qr, false, l, rr);
    F = face_flux<float, FK>(g, f[P_NX * 32], f[P_NY * 32], f[P_A * 32], l, rr, want_lam);
  };
  // flux through the lane's left j-face in row r + 1
  auto jface = [&](const float* s, int r, Flux5<float>& F) {
    const float* f = s + S_JF * 32 + lane;
    float ql[4], qr[4];
    {
      // this cell's state at its right face (the next lane's record), handed to the next lane
      const float cl = f[P_CL * 32 + 1], wlx = f[P_WLX * 32 + 1], wly = f[P_WLY * 32 + 1], sl = f[P_SL * 32 + 1];
      const float cr = f[P_CR * 32], wrx = f[P_WRX * 32], wry = f[P_WRY * 32], sr = f[P_SR * 32];
#pragma unroll
      for (int v = 0; v < 4; ++v) {
        const float gl = fmaf(-dr[v], sl, fmaf(mb[2 * v + 1], wly, mb[2 * v] * wlx));
        const float gr = fmaf(-dl[v], sr, fmaf(mb[2 * v + 1], wry, mb[2 * v] * wrx));
        const float mine = fmaf(cl, strip_limit<LIM>(dr[v], gl), qb[v]);
        ql[v] = __shfl_up_sync(0xffffffffu, mine, 1);
        qr[v] = fmaf(-cr, strip_limit<LIM>(dl[v], gr), qb[v]);
      }
    }
    {
      St<float> l, rr;
      basis_state2(g, ql, qr, false, l, rr);
      F = face_flux<float, FK>(g, f[P_NX * 32], f[P_NY * 32], f[P_A * 32], l, rr, want_lam);
    }
    if (edge_j) {
      // on side 3 the interior cell is the lane to the left; its state is also this lane's
      // (columns past the mesh repeat the last one)
      StripEdge e;
#pragma unroll
      for (int v = 0; v < 8; ++v) {
        const float left = __shfl_up_sync(0xffffffffu, mb[v], 1);
        e.m[v] = jside == 3 ? left : mb[v];
      }
      if (jside >= 0) {
        const bool lo = jside == 2;
#pragma unroll
        for (int v = 0; v < 4; ++v) e.q[v] = qb[v];
        e.nx = f[P_NX * 32]; e.ny = f[P_NY * 32]; e.A = f[P_A * 32];
        e.wx = f[(lo ? P_WRX : P_WLX) * 32]; e.wy = f[(lo ? P_WRY : P_WLY) * 32];
        e.wwx = f[(lo ? P_WLX : P_WRX) * 32]; e.wwy = f[(lo ? P_WLY : P_WRY) * 32];
        strip_edge_flux<FK, LIM>(a, jside, r + 1, e, want_lam, F);
      }
      __syncwarp();
    }
  };
  // move to the next row: r <- r + 1
  auto shift = [&]() {
#pragma unroll
    for (int v = 0; v < 4; ++v) {
      qa[v] = qb[v];
      qb[v] = qc[v];
      qc[v] = qn[v];
    }
#pragma unroll
    for (int v = 0; v < 8; ++v) ma[v] = mb[v];
  };

  const bool sum_in = a.stage > 0;
  const bool update = a.mode == MODE_FUSED_GLOBAL || a.mode == MODE_FUSED_LOCAL;
  const float* sums = a.res_prev[0];
  float rate = 0.f, r2 = 0.f;
  gradient(strip_wait(ring, a.info));
  __syncwarp();
  if (r0 + 1 < r1) fetch_row(r0 + 1, false);
  shift();
#pragma unroll 1
  for (int r = r0 - 1; r < r1; ++r) {
    const float* s = strip_wait(ring, a.info);
    const unsigned cell = unsigned(max(r, 0)) * unsigned(nj) + unsigned(cq);
    gradient(s);
    float jn[4], jnl = 0.f;
#pragma unroll
    for (int v = 0; v < 4; ++v) jn[v] = 0.f;
    if (r + 1 < r1) {
      Flux5<float> F;
      jface(s, r, F);
#pragma unroll
      for (int v = 0; v < 4; ++v) jn[v] = F.f[v] - __shfl_down_sync(0xffffffffu, F.f[v], 1);
      if (want_lam) jnl = F.lam + __shfl_down_sync(0xffffffffu, F.lam, 1);
    }
    // row r + 3 and the update's operands, on their way while the i-face is computed
    float pq[4], ps[4], pl = 0.f;
    {
      const unsigned c3 = qcell(r + 3);
#pragma unroll
      for (int v = 0; v < 4; ++v) {
        qn[v] = (a.q + v * ncell)[c3];
        pq[v] = qa[v];
        ps[v] = 0.f;
      }
    }
    if (update && own && r >= r0) {
      if (a.q0 != a.q) {
#pragma unroll
        for (int v = 0; v < 4; ++v) pq[v] = (a.q0 + v * ncell)[cell];
      }
      if (sum_in) {
#pragma unroll
        for (int v = 0; v < 4; ++v) ps[v] = (sums + v * ncell)[cell];
        if (a.mode == MODE_FUSED_LOCAL) pl = (sums + 4 * ncell)[cell];
      }
    }
    // face-to-cell accumulation (residualCalc.h:199-253 signs)
    float res[4], lam;
    {
      Flux5<float> F;
      iface(s, r, F);
#pragma unroll
      for (int v = 0; v < 4; ++v) {
        res[v] = (fi[v] - F.f[v]) + fj[v];
        fi[v] = F.f[v];
        fj[v] = jn[v];
      }
      lam = (fil + F.lam) + fjl;
      fil = F.lam;
      fjl = jnl;
    }
    const float vol = s[S_VOL * 32 + lane];
    __syncwarp();
    if (r + 3 < r1) fetch_row(r + 3, false);
    if (own && r >= r0) {
      if (a.mode == MODE_RES_MAXRATE || a.mode == MODE_RESIDUAL) {
        if (a.res_out) {
#pragma unroll
          for (int v = 0; v < 4; ++v) (a.res_out + v * ncell)[cell] = res[v];
          (a.res_out + 4 * ncell)[cell] = lam;
        }
        rate = fmaxf(rate, div_near(lam, vol));
        r2 = fmaf(res[2], res[2], r2);
      } else {
        // rungeKuttaAccumulation (timestepping/rungeKutta.h:172-197): the earlier stages'
        // residuals as their sum
        float tot[4];
        const float al = a.alpha[a.stage], ap = a.alpha[0];
        if (sum_in) {
#pragma unroll
          for (int v = 0; v < 4; ++v) {
            tot[v] = fmaf(al, res[v], ap * ps[v]);
            if (a.res_out) (const_cast<float*>(sums) + v * ncell)[cell] = ps[v] + res[v];
          }
        } else {
#pragma unroll
          for (int v = 0; v < 4; ++v) {
            tot[v] = al * res[v];
            if (a.res_out) (a.res_out + v * ncell)[cell] = res[v];
          }
          if (a.res_out) (a.res_out + 4 * ncell)[cell] = lam;
          rate = fmaxf(rate, div_near(lam, vol));
          r2 = fmaf(res[2], res[2], r2);
        }
        float fac;
        if (a.mode == MODE_FUSED_GLOBAL) {
          fac = div_near(a.beta * float(a.info->dt), vol);
        } else {
          // local timestep from the stage-0 spectral radius sum (eulerForwardUpdate.h:155-161)
          const float l0 = sum_in ? pl : lam;
          fac = div_near(a.beta * a.cfl, l0);
        }
        float qo[4];
        forward_update(g, pq, tot, fac, qo, false);
#pragma unroll
        for (int v = 0; v < 4; ++v) (a.q_out + v * ncell)[cell] = qo[v];
        flag_nonphysical(a.info, qo, int(cell));
      }
    }
    shift();
  }
  if (!ring.staged || ring.dead) {
    // after a wait that ran out: the copies still in flight land (bounded again) before the
    // warp's shared memory is given up
    if (ring.dead)
      for (; ring.read < ring.used; ++ring.read) {
        const unsigned k = ring.read % kStripSlots, parity = (ring.read / kStripSlots) & 1u;
        const unsigned long long t0 = globaltimer_ns();
        while (!strip_poll(&ring.bar[k], parity) && globaltimer_ns() - t0 < kCopyWaitNs) {}
      }
    __syncwarp();
  }
  // largest lambda/V and the density-residual norm, once per run
  if (a.mode == MODE_RES_MAXRATE || (a.norm_stage0 && a.stage == 0 && a.mode != MODE_RESIDUAL)) {
    if (a.mode != MODE_FUSED_GLOBAL) {
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) rate = fmaxf(rate, __shfl_xor_sync(0xffffffffu, rate, o));
      if (lane == 0) atomic_max_rate<float>(a.info, rate);
    }
    if (a.norm_stage0) {
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) r2 += __shfl_xor_sync(0xffffffffu, r2, o);
      if (lane == 0) atomicAdd(&a.info->resnorm2, double(r2));
    }
  }
}

// first row of a run
__device__ __forceinline__ int strip_row(int ni, int run, int runs) { return int((long long)ni * run / runs); }

// the warp's ring in the block's shared memory, its barriers initialised
__device__ __forceinline__ StripRing strip_ring(unsigned char* smem, bool staged) {
  const int warp = threadIdx.x >> 5;
  StripRing ring;
  ring.slot = reinterpret_cast<float*>(smem) + size_t(warp) * kStripSlots * kStripRow;
  ring.bar = reinterpret_cast<uint64_t*>(smem + size_t(kStripWarps) * kStripSlots * kStripRow * sizeof(float)) +
             warp * kStripSlots;
  ring.used = ring.read = 0;
  ring.staged = staged;
  ring.dead = false;
  if (staged && (threadIdx.x & 31) == 0) {
    for (int k = 0; k < kStripSlots; ++k) mbar_init(&ring.bar[k], 1);
    mbar_fence_init();
  }
  __syncwarp();
  return ring;
}

template <int FK, int LIM>
__global__ void __launch_bounds__(32 * kStripWarps, 4) strip_kernel(const StripArgs p) {
  extern __shared__ __align__(128) unsigned char smem_raw[];
  const int item = int(blockIdx.x) * kStripWarps + int(threadIdx.x >> 5);
  if (item >= p.strips * p.runs) return;
  if (p.a.clear_words && item == 0 && threadIdx.x == 0) chain_wait<true>();
  clear_step_words(p.a);
  StripRing ring = strip_ring(smem_raw, !p.a.plain_loads);
  const int w = item % p.strips, run = item / p.strips;
  strip_run<FK, LIM>(p.a, p.a.pk, w, strip_row(p.a.ni, run, p.runs), strip_row(p.a.ni, run + 1, p.runs), ring);
}

// The strips of every instance of a batch: the warps of a persistent grid walk the work list
// (b.strip_order, packed instance << 16 | run * strips + strip).  Its launches are not chained:
// a block that starts early while others of the kernel before still run upsets the even split
// of the list (24 meshes, 20 steps from a graph: 12.5 ms chained, 11.4 not).
template <int FK, int LIM>
__global__ void __launch_bounds__(32 * kStripWarps, 4) batch_strip_kernel(const __grid_constant__ BatchArgs<float> b) {
  extern __shared__ __align__(128) unsigned char smem_raw[];
  __shared__ StageArgs<float> sa[kStripWarps];
  const int warp = int(threadIdx.x >> 5), lane = int(threadIdx.x & 31);
  StripRing ring = strip_ring(smem_raw, true);
  for (int i = int(blockIdx.x) * kStripWarps + warp; i < b.strip_work; i += int(gridDim.x) * kStripWarps) {
    const int packed = b.strip_order[i];
    const int k = packed >> 16, t = packed & 0xffff;
    if (lane == 0) sa[warp] = instance_args(b, k);
    __syncwarp();
    const StageArgs<float>& a = sa[warp];
    const int strips = strip_count(a.nj);
    const int w = t % strips, run = t / strips, runs = (a.ni + b.strip_rows - 1) / b.strip_rows;
    strip_run<FK, LIM>(a, a.pk, w, strip_row(a.ni, run, runs), strip_row(a.ni, run + 1, runs), ring);
    __syncwarp();
  }
}

}  // namespace hc
