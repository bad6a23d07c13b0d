// hc_launch.h -- host-side launchers of the per-flux stage kernels.  Each
// flux is compiled in its own translation unit (hc_stage_<flux>.cu) so the
// build runs them in parallel.
#pragma once

#include "hc_kernels.cuh"
#include "hc_stage_warp.cuh"

#include <algorithm>
#include <atomic>
#include <cmath>
#include <limits>
#include <type_traits>
#include <vector>

namespace hc {

// Tile shapes the stage kernel is built for (cells along i x cells along j).
// TILE_16x16_H: 16 x 16 cells run by 128 threads (two cells a thread in the update)
// TILE_AUTO (FP64 single-mesh default): 16x16_H, 8x8 or 4x8 by the mesh's size (f64_auto_tile)
enum TileShape { TILE_8x32 = 0, TILE_4x32 = 1, TILE_16x16 = 2, TILE_16x16_H = 3, TILE_COUNT = 4, TILE_AUTO = 5,
                 TILE_8x8 = 6, TILE_4x8 = 7 };

// SMs of the calling thread's device (asked for once per device)
inline int device_sms() {
  constexpr int kDevices = 64;
  static std::atomic<int> sms[kDevices];
  int dev = 0, n = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) return 152;
  if (dev < kDevices && (n = sms[dev].load(std::memory_order_relaxed)) > 0) return n;
  if (cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || n <= 0) return 152;
  if (dev < kDevices) sms[dev].store(n, std::memory_order_relaxed);
  return n;
}

constexpr int kGridRows = 65535;  // a grid's second dimension: the rows of tiles of a launch

// Tile of an FP64 stage launch.  The stage takes as long as its busiest SM, whose time is the
// FP64 instructions of its tiles: an SM starts one per 19 cycles and each of its four
// sub-partitions one per 64 (measured), whatever the number of active lanes.  So a tile costs
// its warps of faces (230 instructions each), of gradient cells (48) and of cells (60), and
// the shape whose fullest SM is done first wins: small tiles spread a small mesh over the 152
// SMs, large ones repeat fewer faces and gradients.  Measured (Roe, ms per ssp34 step; always
// 16x16 against this rule): 40 x 40 0.263 -> 0.082, 128 x 128 0.260 -> 0.140, 200 x 200 0.394
// -> 0.291; SLAU 300 x 401 0.845 -> 0.649; 256 x 512 and larger stay on 16x16.
inline double f64_tile_cost(int ni, int nj, int ti, int tj, int sms) {
  if ((ni + ti - 1) / ti > kGridRows) return std::numeric_limits<double>::infinity();  // not launchable
  const long long tiles = (long long)((ni + ti - 1) / ti) * ((nj + tj - 1) / tj);
  const double k = double((tiles + sms - 1) / sms);
  auto pass = [k](int items, int instr) {  // warps of one phase, dealt to four sub-partitions
    const double w = k * ((items + 31) / 32);
    return instr * (w > 16 ? 19.0 * w : 64.0 * std::ceil(w / 4));
  };
  return pass((ti + 1) * tj + ti * (tj + 1), 230) + pass((ti + 2) * (tj + 2), 48) + pass(ti * tj, 60);
}
inline int f64_auto_tile(int ni, int nj, int sms = device_sms()) {
  const double c16 = f64_tile_cost(ni, nj, 16, 16, sms), c8 = f64_tile_cost(ni, nj, 8, 8, sms),
               c4 = f64_tile_cost(ni, nj, 4, 8, sms);
  if (c16 <= c8 && c16 <= c4) return TILE_16x16_H;
  return c8 <= c4 ? TILE_8x8 : TILE_4x8;
}

template <class R, int FK> cudaError_t launch_stage(const StageArgs<R>& a, int tile, cudaStream_t s);
template <class R, int FK> cudaError_t prepare_stage();
// persistent batched stage: `grid` CTAs walk the work list of b
template <class R, int FK> cudaError_t launch_batch_stage(const BatchArgs<R>& b, int tile, int grid, cudaStream_t s);

// recording stage (hc_sig_*.cu): one residual evaluation of the 8x32 tile writing the
// face branch signatures to a.sig_i / a.sig_j; DF: double-float stage arithmetic
template <class R, bool DF> cudaError_t launch_sig_stage(const StageArgs<R>& a, int flux, cudaStream_t s);

// one-dimensional path (hc_oned.cu): host geometry of nc cells between nodes x[0..nc]
void oned_geometry(const double* x, int nc, const int bc[2], std::vector<double>& rec, std::vector<double>& vol);

// scalar advection law (hc_stage_scalar.cu): flux is FLUX_RUSANOV or FLUX_CENTRAL
template <class R> cudaError_t prepare_scalar_stage();
template <class R> cudaError_t launch_scalar_stage(const StageArgs<R>& a, int flux, int tile, cudaStream_t s);
template <class R>
cudaError_t launch_scalar_update0(int ni, int nj, const R* q0, const R* res0, const R* vol, R alpha00, R beta0,
                                  double cfl, StepInfo* info, R* q_out, int advance_time, cudaStream_t s);
// residual smoothing of the legacy 1D path (hc_smooth.cu): kind 0 implicit, 1 explicit;
// nplanes planes of n values at `stride`; implicit smoothing needs wrk and tmp of
// nplanes * n values and may run in place (r1 == r0); bc 'p', 'a' or other
template <class R>
cudaError_t launch_smooth_1d(int kind, const R* r0, R* r1, R* wrk, R* tmp, long long n, int nplanes, long long stride,
                             double alpha, int bc, cudaStream_t s);
// batches of scalar-law instances (pools as for the Euler batch)
template <class R>
cudaError_t launch_scalar_batch_stage(const BatchArgs<R>& b, int flux, int tile, int grid, cudaStream_t s);
template <class R>
cudaError_t launch_scalar_batch_update0(const BatchArgs<R>& b, int tile, int grid, double cfl, R alpha00, R beta0,
                                        cudaStream_t s);

// a launch behind the kernel before it on the stream, its blocks waiting in chain_wait
// (chained), or an ordinary one
template <class K, class... A>
inline cudaError_t launch_chained(K* kernel, dim3 grid, unsigned threads, size_t smem, cudaStream_t s, bool chained,
                                  const A&... args) {
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = grid;
  cfg.blockDim = dim3(threads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  cudaLaunchAttribute attr{};
  attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr.val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = &attr;
  cfg.numAttrs = chained ? 1 : 0;
  return cudaLaunchKernelEx(&cfg, kernel, args...);
}

// whether the strip kernel takes an FP32 launch of the 8 x 32 tile: the configuration, and with its
// packed records there
inline bool strips_for(int basis, int limiter) {
  return basis == 0 && (limiter == LIM_VANALBADA || limiter == LIM_VANLEER || limiter == LIM_MINMOD ||
                        limiter == LIM_NOLIMIT2 || limiter == LIM_NOLIMIT3);
}
inline bool strips_take(const float* pk, int basis, int limiter) { return pk && strips_for(basis, limiter); }
// Memory for packed records, after the rest of a mesh's or batch's; null, and the tile kernel takes
// the launches, where there is none left, or (above 256 MiB) they would take more than a quarter of
// what is: 123 bytes a cell on a wide mesh, a fifth of all it needs, but 3,456 a row on a narrow
// one, 1,152 a cell at three columns, which must not cost it the room for its adjoint.
inline cudaError_t alloc_strips(float** pk, size_t bytes) {
  *pk = nullptr;
  if (bytes > (size_t(256) << 20)) {
    size_t free_b = 0, total_b = 0;
    if (cudaError_t e = cudaMemGetInfo(&free_b, &total_b)) return e;
    if (bytes > free_b / 4) return cudaSuccess;
  }
  const cudaError_t e = cudaMalloc((void**)pk, bytes);
  if (e != cudaErrorMemoryAllocation) return e;
  (void)cudaGetLastError();
  *pk = nullptr;
  return cudaSuccess;
}
// the strip kernel's arguments of one mesh
inline StripArgs strip_args(const StageArgs<float>& a) {
  StripArgs p{};
  p.a = a;
  p.strips = strip_count(a.nj);
  p.runs = strip_runs(a.ni, strip_run_rows(1, [&](int) { return a.ni; }, [&](int) { return a.nj; }, device_sms()));
  return p;
}

inline void tile_dims(int tile, int* ti, int* tj) {
  switch (tile) {
    case TILE_4x32: *ti = 4; *tj = 32; break;
    case TILE_16x16:
    case TILE_16x16_H: *ti = 16; *tj = 16; break;
    default: *ti = 8; *tj = 32; break;
  }
}

}  // namespace hc

#define HC_STAGE_INSTANTIATE(FK)                                                                         \
  namespace hc {                                                                                         \
  template <class R, int TI, int TJ> static cudaError_t prep_one() {                                     \
    cudaError_t e = cudaFuncSetAttribute(stage_kernel<TI, TJ, R, FK>,                                    \
                                         cudaFuncAttributeMaxDynamicSharedMemorySize,                    \
                                         int(StageSmem<TI, TJ, R>::bytes));                              \
    if (e != cudaSuccess) return e;                                                                      \
    if (std::is_same<R, double>::value && TI == 8 && TJ == 32) {                                         \
      for (auto kern : {stage_kernel<8, 32, double, FK, df64>, stage_kernel<8, 32, double, FK, df64, 256, LIM_VANALBADA>,\
                        stage_kernel<8, 32, double, FK, df64, 256, LIM_VANLEER>}) {                      \
        e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, int(StageSmem<8, 32, df64>::bytes));\
        if (e != cudaSuccess) return e;                                                                  \
      }                                                                                                  \
    }                                                                                                    \
    return cudaFuncSetAttribute(batch_stage_kernel<TI, TJ, R, FK>,                                       \
                                cudaFuncAttributeMaxDynamicSharedMemorySize,                             \
                                int(StageSmem<TI, TJ, R>::bytes));                                       \
  }                                                                                                      \
  /* FP32, primitive basis, the common limiters: the strip kernel (hc_stage_warp.cuh), with the    */   \
  /* limiter a compile-time constant */                                                                 \
  template <int LIM> static cudaError_t prep_strip() {                                                  \
    cudaError_t e = cudaFuncSetAttribute(strip_kernel<FK, LIM>, cudaFuncAttributeMaxDynamicSharedMemorySize,\
                                         int(kStripSmem));                                              \
    if (e != cudaSuccess) return e;                                                                     \
    return cudaFuncSetAttribute(batch_strip_kernel<FK, LIM>, cudaFuncAttributeMaxDynamicSharedMemorySize,\
                                int(kStripSmem));                                                       \
  }                                                                                                     \
  static cudaError_t prep_strips() {                                                                    \
    cudaError_t e = prep_strip<LIM_VANALBADA>();                                                        \
    if (e == cudaSuccess) e = prep_strip<LIM_VANLEER>();                                                \
    if (e == cudaSuccess) e = prep_strip<LIM_MINMOD>();                                                 \
    if (e == cudaSuccess) e = prep_strip<LIM_NOLIMIT2>();                                               \
    if (e == cudaSuccess) e = prep_strip<LIM_NOLIMIT3>();                                               \
    return e;                                                                                           \
  }                                                                                                     \
  template <int LIM> static bool go_strip(const StageArgs<float>& a, cudaStream_t s) {                  \
    const StripArgs p = strip_args(a);                                                                  \
    const unsigned grid = unsigned((p.strips * p.runs + kStripWarps - 1) / kStripWarps);                \
    launch_chained(strip_kernel<FK, LIM>, dim3(grid), 32 * kStripWarps, kStripSmem, s, a.chained != 0, p); \
    return true;                                                                                        \
  }                                                                                                     \
  static bool go_strips(const StageArgs<float>& a, cudaStream_t s) {                                    \
    if (!strips_take(a.pk, a.basis, a.limiter) || a.dual_src) return false;                             \
    switch (a.limiter) {                                                                                \
      case LIM_VANALBADA: return go_strip<LIM_VANALBADA>(a, s);                                         \
      case LIM_VANLEER: return go_strip<LIM_VANLEER>(a, s);                                             \
      case LIM_MINMOD: return go_strip<LIM_MINMOD>(a, s);                                               \
      case LIM_NOLIMIT2: return go_strip<LIM_NOLIMIT2>(a, s);                                           \
      case LIM_NOLIMIT3: return go_strip<LIM_NOLIMIT3>(a, s);                                           \
      default: return false;                                                                            \
    }                                                                                                   \
  }                                                                                                     \
  /* What the strips leave to the FP32 8x32 tile (the conserved basis, dual time, no packed  */        \
  /* records), with the common limiters compile-time constants: 256 x 512, 20 steps, SLAU +  */        \
  /* van Leer, conserved 1.37 ms chosen at run time, 1.15 so; dual time 1.58 and 1.36       */         \
  template <int LIM> static bool go_lim(const StageArgs<float>& a, cudaStream_t s) {                   \
    const dim3 grid((a.nj + 31) / 32, (a.ni + 7) / 8);                                                 \
    launch_chained(stage_kernel<8, 32, float, FK, float, 256, LIM>, grid, 256, StageSmem<8, 32, float>::bytes, s, \
                   a.chained != 0, a);                                                                 \
    return true;                                                                                       \
  }                                                                                                    \
  static bool go_lims(const StageArgs<float>& a, cudaStream_t s) {                                     \
    switch (a.limiter) {                                                                               \
      case LIM_VANALBADA: return go_lim<LIM_VANALBADA>(a, s);                                          \
      case LIM_VANLEER: return go_lim<LIM_VANLEER>(a, s);                                              \
      case LIM_MINMOD: return go_lim<LIM_MINMOD>(a, s);                                                \
      case LIM_NOLIMIT2: return go_lim<LIM_NOLIMIT2>(a, s);                                            \
      case LIM_NOLIMIT3: return go_lim<LIM_NOLIMIT3>(a, s);                                            \
      default: return false;                                                                           \
    }                                                                                                  \
  }                                                                                                    \
  template <int LIM> static bool gob_strip(const BatchArgs<float>& b, cudaStream_t s) {                 \
    batch_strip_kernel<FK, LIM><<<unsigned(b.strip_grid), 32 * kStripWarps, kStripSmem, s>>>(b);        \
    return true;                                                                                        \
  }                                                                                                     \
  static bool gob_strips(const BatchArgs<float>& b, cudaStream_t s) {                                   \
    if (!strips_take(b.pk, b.basis, b.limiter)) return false;                                           \
    switch (b.limiter) {                                                                                \
      case LIM_VANALBADA: return gob_strip<LIM_VANALBADA>(b, s);                                        \
      case LIM_VANLEER: return gob_strip<LIM_VANLEER>(b, s);                                            \
      case LIM_MINMOD: return gob_strip<LIM_MINMOD>(b, s);                                              \
      case LIM_NOLIMIT2: return gob_strip<LIM_NOLIMIT2>(b, s);                                          \
      case LIM_NOLIMIT3: return gob_strip<LIM_NOLIMIT3>(b, s);                                          \
      default: return false;                                                                            \
    }                                                                                                   \
  }                                                                                                     \
  template <class R, int TI, int TJ, int LIM = -1>                                                        \
  static void gob(const BatchArgs<R>& b, int grid, cudaStream_t s) {                                     \
    /* a persistent grid larger than what stays resident would run a second, partial wave */           \
    static int cap = 0;                                                                                  \
    if (cap == 0) {                                                                                      \
      int dev = 0, sms = 0, occ = 0;                                                                     \
      cudaGetDevice(&dev);                                                                               \
      cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);                                 \
      cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, batch_stage_kernel<TI, TJ, R, FK, LIM>, TI * TJ, \
                                                    StageSmem<TI, TJ, R>::bytes);                        \
      cap = (sms > 0 && occ > 0) ? sms * occ : grid;                                                     \
    }                                                                                                    \
    batch_stage_kernel<TI, TJ, R, FK, LIM><<<std::min(grid, cap), TI * TJ, StageSmem<TI, TJ, R>::bytes, s>>>( \
        b);                                                                                              \
  }                                                                                                      \
  template <int LIM> static void gob_tile(const BatchArgs<float>& b, int tile, int grid, cudaStream_t s) { \
    if (tile == TILE_4x32) gob<float, 4, 32, LIM>(b, grid, s);                                           \
    else if (tile == TILE_16x16) gob<float, 16, 16, LIM>(b, grid, s);                                    \
    else gob<float, 8, 32, LIM>(b, grid, s);                                                             \
  }                                                                                                      \
  template <> cudaError_t launch_batch_stage<double, FK>(const BatchArgs<double>& b, int tile, int grid, \
                                                         cudaStream_t s) {                               \
    if (tile == TILE_4x32) gob<double, 4, 32>(b, grid, s);                                               \
    else if (tile == TILE_16x16) gob<double, 16, 16>(b, grid, s);                                        \
    else gob<double, 8, 32>(b, grid, s);                                                                 \
    return cudaGetLastError();                                                                           \
  }                                                                                                      \
  template <> cudaError_t launch_batch_stage<float, FK>(const BatchArgs<float>& b, int tile, int grid,   \
                                                        cudaStream_t s) {                                \
    if (tile == TILE_8x32 && gob_strips(b, s)) return cudaGetLastError();                                \
    if (b.limiter == LIM_VANALBADA) gob_tile<LIM_VANALBADA>(b, tile, grid, s);                           \
    else if (b.limiter == LIM_NOLIMIT3) gob_tile<LIM_NOLIMIT3>(b, tile, grid, s);                        \
    else gob_tile<-1>(b, tile, grid, s);                                                                 \
    return cudaGetLastError();                                                                           \
  }                                                                                                      \
  template <class R, int TI, int TJ> static void go(const StageArgs<R>& a, cudaStream_t s) {             \
    const dim3 grid((a.nj + TJ - 1) / TJ, (a.ni + TI - 1) / TI);                                         \
    launch_chained(stage_kernel<TI, TJ, R, FK>, grid, TI * TJ, StageSmem<TI, TJ, R>::bytes, s,           \
                   a.chained != 0, a);                                                                   \
  }                                                                                                      \
  template <class R> static cudaError_t prep_half() {                                                   \
    return cudaFuncSetAttribute(stage_kernel<16, 16, R, FK, R, 128>,                                     \
                                cudaFuncAttributeMaxDynamicSharedMemorySize,                             \
                                int(StageSmem<16, 16, R>::bytes));                                       \
  }                                                                                                      \
  template <> cudaError_t prepare_stage<double, FK>() {                                                  \
    cudaError_t e = prep_one<double, 8, 32>();                                                           \
    if (e == cudaSuccess) e = prep_one<double, 4, 32>();                                                 \
    if (e == cudaSuccess) e = prep_one<double, 16, 16>();                                                \
    if (e == cudaSuccess) e = prep_half<double>();                                                       \
    return e;                                                                                            \
  }                                                                                                      \
  template <> cudaError_t prepare_stage<float, FK>() {                                                   \
    cudaError_t e = prep_one<float, 8, 32>();                                                            \
    if (e == cudaSuccess) e = prep_one<float, 4, 32>();                                                  \
    if (e == cudaSuccess) e = prep_one<float, 16, 16>();                                                 \
    if (e == cudaSuccess) e = prep_half<float>();                                                        \
    if (e == cudaSuccess) e = prep_strips();                                                             \
    return e;                                                                                            \
  }                                                                                                      \
  template <class R> static cudaError_t dispatch(const StageArgs<R>& a, int tile, cudaStream_t s) {     \
    if (std::is_same<R, double>::value && a.fic) {                                                       \
      /* Double-float compute type, 8x32 tiles.  The two limiters with a packed form are compile-time */ \
      /* constants: the selection among ten, four variables a face, keeps their code from overlapping */ \
      /* (512 x 1024, van Albada, a step: 0.91 ms chosen at run time, 0.81 so) */                        \
      const dim3 grid((a.nj + 31) / 32, (a.ni + 7) / 8);                                                 \
      const auto kern = a.limiter == LIM_VANALBADA ? stage_kernel<8, 32, double, FK, df64, 256, LIM_VANALBADA>\
                        : a.limiter == LIM_VANLEER ? stage_kernel<8, 32, double, FK, df64, 256, LIM_VANLEER>\
                                                   : stage_kernel<8, 32, double, FK, df64>;              \
      return launch_chained(kern, grid, 256, StageSmem<8, 32, df64>::bytes, s, a.chained != 0,           \
                            *reinterpret_cast<const StageArgs<double>*>(&a));                            \
    }                                                                                                    \
    if constexpr (std::is_same<R, float>::value) {                                                       \
      if ((tile == TILE_8x32 || tile < 0 || tile >= TILE_COUNT) && (go_strips(a, s) || go_lims(a, s)))   \
        return cudaGetLastError();                                                                       \
    }                                                                                                    \
    if constexpr (std::is_same<R, double>::value) {                                                      \
      if (tile == TILE_AUTO) tile = f64_auto_tile(a.ni, a.nj);                                           \
      if (tile == TILE_8x8) {                                                                            \
        const dim3 grid((a.nj + 7) / 8, (a.ni + 7) / 8);                                                 \
        return launch_chained(stage_kernel<8, 8, R, FK, R, 160>, grid, 160, StageSmem<8, 8, R>::bytes, s, \
                              a.chained != 0, a);                                                        \
      }                                                                                                  \
      if (tile == TILE_4x8) {                                                                            \
        const dim3 grid((a.nj + 7) / 8, (a.ni + 3) / 4);                                                 \
        return launch_chained(stage_kernel<4, 8, R, FK, R, 96>, grid, 96, StageSmem<4, 8, R>::bytes, s,  \
                              a.chained != 0, a);                                                        \
      }                                                                                                  \
    }                                                                                                    \
    if (tile == TILE_4x32) go<R, 4, 32>(a, s);                                                           \
    else if (tile == TILE_16x16) go<R, 16, 16>(a, s);                                                    \
    else if (tile == TILE_16x16_H) {                                                                     \
      const dim3 grid((a.nj + 15) / 16, (a.ni + 15) / 16);                                               \
      return launch_chained(stage_kernel<16, 16, R, FK, R, 128>, grid, 128, StageSmem<16, 16, R>::bytes, s, \
                            a.chained != 0, a);                                                          \
    } else go<R, 8, 32>(a, s);                                                                           \
    return cudaGetLastError();                                                                           \
  }                                                                                                      \
  template <> cudaError_t launch_stage<double, FK>(const StageArgs<double>& a, int tile, cudaStream_t s) { \
    return dispatch<double>(a, tile, s);                                                                 \
  }                                                                                                      \
  template <> cudaError_t launch_stage<float, FK>(const StageArgs<float>& a, int tile, cudaStream_t s) {   \
    return dispatch<float>(a, tile, s);                                                                  \
  }                                                                                                      \
  }
