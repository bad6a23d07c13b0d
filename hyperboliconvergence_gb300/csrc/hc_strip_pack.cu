// hc_strip_pack.cu -- the face records of a mesh in the layout of the FP32 strip kernel
// (hc_stage_warp.cuh), built once per mesh from the FP64 records.
#include "hc_stage_warp.cuh"

namespace hc {

__global__ void pack_strips_kernel(const double* __restrict__ fi, const double* __restrict__ fj,
                                   const double* __restrict__ vol, int ni, int nj, int per_i, int per_j,
                                   float* __restrict__ out) {
  const int rows = ni + kStripRowsBefore;
  const size_t total = size_t(strip_count(nj)) * rows * 32;
  const size_t nfi = size_t(ni + 1) * nj, nfj = size_t(ni) * (nj + 1);
  for (size_t k = blockIdx.x * size_t(blockDim.x) + threadIdx.x; k < total; k += size_t(gridDim.x) * blockDim.x) {
    const int lane = int(k % 32);
    const int r = int((k / 32) % rows) - kStripRowsBefore, w = int(k / 32 / rows);
    const int c = w * kStripCells - 2 + lane;
    const int cc = per_j ? wrapi(c, nj) : min(max(c, 0), nj - 1);      // column of cells and i-faces
    const int cf = per_j ? wrapi(c, nj) : min(max(c, 0), nj);          // its left j-face
    const bool in_c = per_j || (c >= 0 && c <= nj);
    auto row_cell = [&](int i) { return per_i ? wrapi(i, ni) : min(max(i, 0), ni - 1); };
    auto row_face = [&](int i) { return per_i ? wrapi(i, ni) : min(max(i, 0), ni); };
    auto in_row = [&](int i, int n) { return per_i || (i >= 0 && i < n); };
    float* o = out + (size_t(w) * rows + (r + kStripRowsBefore)) * kStripRow + lane;
    auto put = [&](int f, double v) { o[f * 32] = float(v); };
    {  // the gradient sums of row r + 1
      const size_t f = size_t(row_cell(r + 1)) * (nj + 1) + cf;
      const bool ok = in_c && in_row(r + 1, ni);
      put(S_DXJ, ok ? fj[F_DXX * nfj + f] : 0.);
      put(S_DXJ + 1, ok ? fj[F_DXY * nfj + f] : 0.);
      const size_t g = size_t(row_face(r + 2)) * nj + cc;
      const bool oi = in_row(r + 2, ni + 1);
      put(S_DXI, oi ? fi[F_DXX * nfi + g] : 0.);
      put(S_DXI + 1, oi ? fi[F_DXY * nfi + g] : 0.);
    }
    // a face: its limiter weights scaled by dl + dr; on a boundary face the interior side's,
    // with half the (mirrored) distance, and the wall extrapolation weights as they are
    auto face = [&](int base, const double* rec, size_t nf, size_t f, int side) {
      const double dl = rec[F_DL * nf + f], dr = rec[F_DR * nf + f], d = dl + dr;
      put(base + P_NX, rec[F_NX * nf + f]);
      put(base + P_NY, rec[F_NY * nf + f]);
      put(base + P_A, rec[F_A * nf + f]);
      put(base + P_CL, dl / d);
      put(base + P_CR, dr / d);
      const double sl = side == 0 ? 1. : d, sr = side == 1 ? 1. : d;  // side 0: low boundary, 1: high
      put(base + P_WLX, rec[F_WLX * nf + f] * sl);
      put(base + P_WLY, rec[F_WLY * nf + f] * sl);
      put(base + P_SL, rec[F_SL * nf + f] * sl);
      put(base + P_WRX, rec[F_WRX * nf + f] * sr);
      put(base + P_WRY, rec[F_WRY * nf + f] * sr);
      put(base + P_SR, rec[F_SR * nf + f] * sr);
    };
    {
      const int i = row_face(r + 1);
      face(S_IF, fi, nfi, size_t(i) * nj + cc, per_i ? -1 : (i == 0 ? 0 : (i == ni ? 1 : -1)));
    }
    put(S_VOL, vol[size_t(row_cell(r)) * nj + cc]);
    face(S_JF, fj, nfj, size_t(row_cell(r + 1)) * (nj + 1) + cf, per_j ? -1 : (cf == 0 ? 0 : (cf == nj ? 1 : -1)));
  }
}

cudaError_t pack_strips(const double* fi, const double* fj, const double* vol, int ni, int nj, const int bc[4],
                        float* out, cudaStream_t s) {
  const size_t total = size_t(strip_count(nj)) * (ni + kStripRowsBefore) * 32;
  pack_strips_kernel<<<unsigned(std::min<size_t>((total + 255) / 256, 152 * 32)), 256, 0, s>>>(
      fi, fj, vol, ni, nj, bc[0] == BC_PERIODIC, bc[2] == BC_PERIODIC, out);
  return cudaGetLastError();
}

}  // namespace hc
