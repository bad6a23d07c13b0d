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
// -s (dl + dr), dl/(dl + dr) and -dr/(dl + dr): the limiters are homogeneous, and the division
// by that distance disappears.
//
// What bounds it: instruction issue (58% of the issue slots at four warps per scheduler, FMA 30%, no
// other pipe above 26%; 845 instructions per warp and row).  So what comes in twos -- a face's left and
// right side, a gradient's x and y -- is computed as packed FP32 pairs, one instruction for two
// operations, from records that hold the pairs side by side, and the planes are addressed by a
// 32-bit byte offset that serves all of them: 912 instructions before and 834 with the pairs (the
// waits' votes and the roots' selections came later), 512 x 1024 O-grid, Roe + van Albada: 0.104 ->
// 0.096 ms per ssp34 step (0.097 now), 301 x 715, AUSM+up + van Leer: 0.062 -> 0.059.
// The tiled kernel before the strips (8 x 32 cells, halo and gradient tiles in shared memory,
// four block barriers) issued a third more at 45%, waiting on barriers and on the j-face records:
// 0.174 and 0.100 ms; a batch of 24 uneven quadrant problems, SLAU, 20 steps, uploads and downloads
// included: 18.8 ms, now 14.2 (with the update's launch, hc_batch.h).
// Four blocks of four warps per SM: at most 128 registers, which hold a pass without spills (with
// the edge faces' code out of line the calls cost 48 bytes of spills and 15% of the time), and
// 512 x 1024 in runs of 8 rows is one wave of 2,368 warps.
//
// The stage residuals of the alpha/beta tables are kept as their running sum (each row of every
// table weighs the earlier stages alike, ode.h:107-197), so a later stage reads and writes one
// 4-plane buffer whatever its number.
#pragma once

#include "hc_kernels.cuh"
#include "hc_pair.cuh"

#include <algorithm>
#include <cmath>

namespace hc {

constexpr int kStripCells = 28;                      // columns a strip owns
constexpr int kStripRowsBefore = 3;                  // record rows before row 0 (the run's lead-in)
// A record row r, in units of 32 floats and in the order of the first and last rows' needs: the
// gradient sums of row r + 1 (left j-face and lower i-face offsets), the i-face r + 1, the
// volume of row r, the j-face on the left of row r + 1.
enum StripField { S_DXJ = 0, S_DXI = 2, S_IF = 4, S_VOL = 15, S_JF = 16, S_FIELDS = 27 };
// Fields of a face within S_IF / S_JF, likewise.  All but the area are pairs, a lane's two
// values side by side: the weights of the face's left and right side (of a j-face: of the cell's
// right face as its left side, and of its left face as its right side, so that both are the
// lane's own cell's), the sums' factors -s and the distances cl, -cr alike, and the normal.
enum StripFace { P_WX = 0, P_WY = 2, P_S = 4, P_C = 6, P_N = 8, P_A = 10, P_FIELDS = 11 };
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
// 1024 with 8 rows (one wave) 0.104, with 16 (half a wave: each warp's latency is exposed) 0.21;
// a batch of 24 meshes, 2.27 M cells, with 8 rows (4.2 waves) 0.64, by this rule (2 waves) 0.57;
// 96 small ones, 0.47 M cells, 0.255 and 0.20.
inline int strip_runs(int ni, int rows) { return (ni + rows - 1) / rows; }
// most: the work items that a mesh may have (0: any number); 0 is returned where a mesh has more
// whatever the rows.
template <class NI, class NJ> inline int strip_run_rows(int n, NI ni, NJ nj, int sms, long long most = 0) {
  constexpr int kResident = 16;  // warps per SM
  int best = 0;
  double cost = 1e300;
  for (int rows = 1; rows <= 64; ++rows) {
    long long items = 0;
    int longest = 0;
    bool fits = true;
    for (int k = 0; k < n; ++k) {
      const int runs = strip_runs(ni(k), rows);
      const long long m = (long long)strip_count(nj(k)) * runs;
      items += m;
      longest = std::max(longest, (ni(k) + runs - 1) / runs);
      fits = fits && (most == 0 || m <= most);
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

// Value at a byte offset of 32 bits from a plane's base (the same in every lane, so that one
// address register serves all planes).
__device__ __forceinline__ float at(const float* plane, unsigned off) {
  return *reinterpret_cast<const float*>(reinterpret_cast<const char*>(plane) + off);
}
__device__ __forceinline__ float& at(float* plane, unsigned off) {
  return *reinterpret_cast<float*>(reinterpret_cast<char*>(plane) + off);
}
// a lane's pair of a record field
__device__ __forceinline__ f2 pair_at(const float* p) {
  f2 r;
  r.v = *reinterpret_cast<const unsigned long long*>(p);
  return r;
}

// ---- limiters on arguments scaled by the centres' distance
template <int LIM> __device__ __forceinline__ float strip_limit(float a, float b) {
  if constexpr (LIM == LIM_VANALBADA) {
    const float ab = fmaxf(a * b, 0.f);  // 0 slope where a b <= 0; a NaN comes back with a + b
    return (ab * (a + b)) * rcp_f32(fmaf(b, b, fmaf(a, a, FLT_MIN)));
  } else if constexpr (LIM == LIM_VANLEER) {
    const float ab = a * b;
    const float s = (ab + ab) * rcp_f32(a + b);
    return ab <= 0.f ? 0.f : s;
  } else {
    return limit<float>(LIM, a, b);
  }
}
template <int LIM> __device__ __forceinline__ f2 strip_limit2(f2 a, f2 b) {
  if constexpr (LIM == LIM_VANALBADA) {
    const f2 t = mul2(a, b);
    const f2 ab = pair(fmaxf(lo(t), 0.f), fmaxf(hi(t), 0.f));
    const f2 den = fma2(b, b, fma2(a, a, pair(FLT_MIN, FLT_MIN)));
    return mul2(mul2(ab, add2(a, b)), pair(rcp_f32(lo(den)), rcp_f32(hi(den))));
  } else if constexpr (LIM == LIM_VANLEER) {
    const f2 ab = mul2(a, b), sum = add2(a, b);
    const f2 s = mul2(add2(ab, ab), pair(rcp_f32(lo(sum)), rcp_f32(hi(sum))));
    return pair(lo(ab) <= 0.f ? 0.f : lo(s), hi(ab) <= 0.f ? 0.f : hi(s));
  } else {
    return pair(strip_limit<LIM>(lo(a), lo(b)), strip_limit<LIM>(hi(a), hi(b)));
  }
}
// the two states of a face from the pairs {left, right} of its primitive values (prim_state_ir)
__device__ __forceinline__ void strip_states(const Gas<float>& g, const f2* q, St<float>& l, St<float>& r) {
  const f2 ir = pair(rcp_f32(lo(q[2])), rcp_f32(hi(q[2])));
  const f2 u2 = fma2(q[1], q[1], mul2(q[0], q[0]));
  const f2 a2 = mul2(pair(g.gamma, g.gamma), mul2(q[3], ir));
  const f2 h = fma2(a2, pair(g.gamma1, g.gamma1), mul2(pair(0.5f, 0.5f), u2));
  l.u = lo(q[0]); l.v = lo(q[1]); l.r = lo(q[2]); l.p = lo(q[3]);
  l.u2 = lo(u2); l.ir = lo(ir); l.a2 = lo(a2); l.h = lo(h);
  r.u = hi(q[0]); r.v = hi(q[1]); r.r = hi(q[2]); r.p = hi(q[3]);
  r.u2 = hi(u2); r.ir = hi(ir); r.a2 = hi(a2); r.h = hi(h);
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
// Whether the copy of fetch k has landed, waiting for it at most kCopyWaitNs.  The lanes' polls may
// differ, so the warp goes by their vote: one answer, which every lane acts on together.
__device__ __forceinline__ bool strip_landed(const StripRing& ring, unsigned k) {
  constexpr unsigned all = 0xffffffffu;
  uint64_t* bar = &ring.bar[k % kStripSlots];
  const unsigned parity = (k / kStripSlots) & 1u;
  if (__all_sync(all, strip_poll(bar, parity))) return true;
  const unsigned long long t0 = globaltimer_ns();
  for (;;) {
    const bool late = __any_sync(all, globaltimer_ns() - t0 > kCopyWaitNs);
    if (__all_sync(all, strip_poll(bar, parity))) return true;
    if (late) return false;
  }
}
// wait for the next fetched row (at most kCopyWaitNs) and return its slot
__device__ __forceinline__ const float* strip_wait(StripRing& ring, StepInfo* info) {
  const unsigned k = ring.read;
  if (ring.staged && !ring.dead && !strip_landed(ring, k)) {
    ring.dead = true;  // no further copies or waits; the rows computed from here are discarded with the step
    atomicCAS(&info->status, ST_OK, ST_TIMEOUT);
    // what is still in flight, this row's copy too, lands (each waited for again, bounded) before
    // anything else may become of the warp's shared memory
    for (unsigned f = k; f != ring.used; ++f) (void)strip_landed(ring, f);
  }
  if (!ring.dead) ring.read = k + 1;  // a dead ring stays at the row that failed
  __syncwarp();
  return ring.slot + (k % kStripSlots) * kStripRow;
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
  // byte offset of the lane's cell in row r (fewer than 2^28 cells)
  auto qcell = [&](int r) -> unsigned {
    int rr = r;
    if (per_i) { if (rr < 0 || rr >= ni) rr = wrapi(rr, ni); }
    else rr = min(max(rr, 0), ni - 1);
    return (unsigned(rr) * unsigned(nj) + unsigned(cq)) * 4u;
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
      qa[v] = at(p, k0);
      qb[v] = at(p, k1);
      qc[v] = at(p, k2);
      qn[v] = at(p, k3);
    }
  }
  // offset {x, y} of the i-face between rows r and r + 1
  f2 di = pair_at(recrow(r0 - 3) + S_DXI * 32 + 2 * lane);
  f2 mx[4], my[4];      // gradient sums {of row r, of row r + 1}, x and y
  float dl[4], dr[4];   // jumps over the left and right faces in row r + 1
  float fi[4], fil = 0.f;  // flux through the i-face r (the upper face of row r)
  float fj[4], fjl = 0.f;  // net j-flux of row r
#pragma unroll
  for (int v = 0; v < 4; ++v) { fi[v] = fj[v] = 0.f; mx[v] = my[v] = pair(0.f, 0.f); }

  // gradient sums (lsq/qmetric.ipp) of row r + 1 from rows r, r + 1, r + 2
  auto gradient = [&](const float* s) {
    const f2 dj0 = pair_at(s + S_DXJ * 32 + 2 * lane), dj1 = pair_at(s + S_DXJ * 32 + 2 * lane + 2);
    const f2 di1 = pair_at(s + S_DXI * 32 + 2 * lane);
#pragma unroll
    for (int v = 0; v < 4; ++v) {
      const float left = __shfl_up_sync(0xffffffffu, qb[v], 1);
      dl[v] = qb[v] - left;
      dr[v] = __shfl_down_sync(0xffffffffu, dl[v], 1);
      const float a0 = qb[v] - qa[v], a1 = qc[v] - qb[v];
      const f2 m = fma2(pair(dr[v], dr[v]), dj1,
                        fma2(pair(dl[v], dl[v]), dj0, fma2(pair(a1, a1), di1, mul2(pair(a0, a0), di))));
      mx[v] = pair(lo(mx[v]), lo(m));
      my[v] = pair(lo(my[v]), hi(m));
    }
    di = di1;
  };
  // flux through the i-face r + 1, between rows r and r + 1
  auto iface = [&](const float* s, int r, Flux5<float>& F) {
    const float* f = s + S_IF * 32 + 2 * lane;
    const int face = r + 1;
    const f2 n = pair_at(f + P_N * 32);
    const float area = s[(S_IF + P_A) * 32 + lane];
    if (!per_i && (face == 0 || face == ni)) {
      const bool low = face == 0;
      StripEdge e;
#pragma unroll
      for (int v = 0; v < 4; ++v) {
        e.q[v] = low ? qb[v] : qa[v];
        e.m[2 * v] = low ? hi(mx[v]) : lo(mx[v]);
        e.m[2 * v + 1] = low ? hi(my[v]) : lo(my[v]);
      }
      e.nx = lo(n); e.ny = hi(n); e.A = area;
      const f2 wx = pair_at(f + P_WX * 32), wy = pair_at(f + P_WY * 32);
      e.wx = low ? hi(wx) : lo(wx); e.wy = low ? hi(wy) : lo(wy);
      e.wwx = low ? lo(wx) : hi(wx); e.wwy = low ? lo(wy) : hi(wy);
      strip_edge_flux<FK, LIM>(a, low ? 0 : 1, cq, e, want_lam, F);
      return;
    }
    f2 q[4];  // {left, right}
    {
      const f2 wx = pair_at(f + P_WX * 32), wy = pair_at(f + P_WY * 32), ns = pair_at(f + P_S * 32),
               c = pair_at(f + P_C * 32);
#pragma unroll
      for (int v = 0; v < 4; ++v) {
        const float d = qb[v] - qa[v];
        const f2 dq = pair(d, d);
        const f2 gr = fma2(dq, ns, fma2(my[v], wy, mul2(mx[v], wx)));
        q[v] = fma2(c, strip_limit2<LIM>(dq, gr), pair(qa[v], qb[v]));
      }
    }
    St<float> l, rr;
    strip_states(g, q, l, rr);
    F = face_flux<float, FK>(g, lo(n), hi(n), area, l, rr, want_lam);
  };
  // flux through the lane's left j-face in row r + 1
  auto jface = [&](const float* s, int r, Flux5<float>& F) {
    const float* f = s + S_JF * 32 + 2 * lane;
    const f2 n = pair_at(f + P_N * 32);
    const float area = s[(S_JF + P_A) * 32 + lane];
    f2 q[4];  // {left, right}
    {
      // this cell's states at its right face, handed to the next lane, and at its left face
      const f2 wx = pair_at(f + P_WX * 32), wy = pair_at(f + P_WY * 32), ns = pair_at(f + P_S * 32),
               c = pair_at(f + P_C * 32);
#pragma unroll
      for (int v = 0; v < 4; ++v) {
        const f2 dq = pair(dr[v], dl[v]);
        const f2 gr = fma2(dq, ns, fma2(pair(hi(my[v]), hi(my[v])), wy, mul2(pair(hi(mx[v]), hi(mx[v])), wx)));
        const f2 x = fma2(c, strip_limit2<LIM>(dq, gr), pair(qb[v], qb[v]));
        q[v] = pair(__shfl_up_sync(0xffffffffu, lo(x), 1), hi(x));
      }
    }
    {
      St<float> l, rr;
      strip_states(g, q, l, rr);
      F = face_flux<float, FK>(g, lo(n), hi(n), area, l, rr, want_lam);
    }
    if (edge_j) {
      // on side 3 the interior cell is the lane to the left; its state is also this lane's
      // (columns past the mesh repeat the last one)
      StripEdge e;
#pragma unroll
      for (int v = 0; v < 4; ++v) {
        const float x = hi(mx[v]), y = hi(my[v]);
        const float xl = __shfl_up_sync(0xffffffffu, x, 1), yl = __shfl_up_sync(0xffffffffu, y, 1);
        e.m[2 * v] = jside == 3 ? xl : x;
        e.m[2 * v + 1] = jside == 3 ? yl : y;
      }
      if (jside >= 0) {
        const bool low = jside == 2;
#pragma unroll
        for (int v = 0; v < 4; ++v) e.q[v] = qb[v];
        e.nx = lo(n); e.ny = hi(n); e.A = area;
        // the left face's weights: its left side's in the pair of the lane before
        const float wlx = f[P_WX * 32 - 2], wly = f[P_WY * 32 - 2];
        const float wrx = f[P_WX * 32 + 1], wry = f[P_WY * 32 + 1];
        e.wx = low ? wrx : wlx; e.wy = low ? wry : wly;
        e.wwx = low ? wlx : wrx; e.wwy = low ? wly : wry;
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
    for (int v = 0; v < 4; ++v) {
      mx[v] = pair(hi(mx[v]), hi(mx[v]));
      my[v] = pair(hi(my[v]), hi(my[v]));
    }
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
    const unsigned cell = (unsigned(max(r, 0)) * unsigned(nj) + unsigned(cq)) * 4u;
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
        qn[v] = at(a.q + v * ncell, c3);
        pq[v] = qa[v];
        ps[v] = 0.f;
      }
    }
    if (update && own && r >= r0) {
      if (a.q0 != a.q) {
#pragma unroll
        for (int v = 0; v < 4; ++v) pq[v] = at(a.q0 + v * ncell, cell);
      }
      if (sum_in) {
#pragma unroll
        for (int v = 0; v < 4; ++v) ps[v] = at(sums + v * ncell, cell);
        if (a.mode == MODE_FUSED_LOCAL) pl = at(sums + 4 * ncell, cell);
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
          for (int v = 0; v < 4; ++v) at(a.res_out + v * ncell, cell) = res[v];
          at(a.res_out + 4 * ncell, cell) = lam;
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
            if (a.res_out) at(const_cast<float*>(sums) + v * ncell, cell) = ps[v] + res[v];
          }
        } else {
#pragma unroll
          for (int v = 0; v < 4; ++v) {
            tot[v] = al * res[v];
            if (a.res_out) at(a.res_out + v * ncell, cell) = res[v];
          }
          if (a.res_out) at(a.res_out + 4 * ncell, cell) = lam;
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
        for (int v = 0; v < 4; ++v) at(a.q_out + v * ncell, cell) = qo[v];
        flag_nonphysical(a.info, qo, int(cell / 4u));
      }
    }
    shift();
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
    if (ring.dead) {  // a copy of an earlier item never landed: this one cannot be computed either
      if (lane == 0) atomicCAS(&b.info[k].status, ST_OK, ST_TIMEOUT);
      continue;
    }
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
