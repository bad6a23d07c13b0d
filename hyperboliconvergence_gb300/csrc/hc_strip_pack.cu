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
    float* o = out + (size_t(w) * rows + (r + kStripRowsBefore)) * kStripRow;
    auto put = [&](int f, double v) { o[f * 32 + lane] = float(v); };
    auto put2 = [&](int f, double x, double y) { o[f * 32 + 2 * lane] = float(x); o[f * 32 + 2 * lane + 1] = float(y); };
    {  // the gradient sums of row r + 1
      const size_t f = size_t(row_cell(r + 1)) * (nj + 1) + cf;
      const bool ok = in_c && in_row(r + 1, ni);
      put2(S_DXJ, ok ? fj[F_DXX * nfj + f] : 0., ok ? fj[F_DXY * nfj + f] : 0.);
      const size_t g = size_t(row_face(r + 2)) * nj + cc;
      const bool oi = in_row(r + 2, ni + 1);
      put2(S_DXI, oi ? fi[F_DXX * nfi + g] : 0., oi ? fi[F_DXY * nfi + g] : 0.);
    }
    // A face: the limiter weights of its left side (of face fl) and of its right side (of face fr;
    // the same for an i-face) scaled by dl + dr; on a boundary face the interior side's, with
    // half the (mirrored) distance, and the wall extrapolation weights as they are.  side: 0 the
    // low boundary's face, 1 the high one's, -1 neither.
    auto face = [&](int base, const double* rec, size_t nf, size_t fl, int side_l, size_t fr, int side_r) {
      const double dl = rec[F_DL * nf + fl] + rec[F_DR * nf + fl], dr = rec[F_DL * nf + fr] + rec[F_DR * nf + fr];
      const double sl = side_l == 0 ? 1. : dl, sr = side_r == 1 ? 1. : dr;
      put2(base + P_WX, rec[F_WLX * nf + fl] * sl, rec[F_WRX * nf + fr] * sr);
      put2(base + P_WY, rec[F_WLY * nf + fl] * sl, rec[F_WRY * nf + fr] * sr);
      put2(base + P_S, -(rec[F_SL * nf + fl] * sl), -(rec[F_SR * nf + fr] * sr));
      put2(base + P_C, rec[F_DL * nf + fl] / dl, -(rec[F_DR * nf + fr] / dr));
      put2(base + P_N, rec[F_NX * nf + fr], rec[F_NY * nf + fr]);
      put(base + P_A, rec[F_A * nf + fr]);
    };
    {
      const int i = row_face(r + 1);
      const size_t f = size_t(i) * nj + cc;
      const int side = per_i ? -1 : (i == 0 ? 0 : (i == ni ? 1 : -1));
      face(S_IF, fi, nfi, f, side, f, side);
    }
    put(S_VOL, vol[size_t(row_cell(r)) * nj + cc]);
    {
      const int cr = per_j ? wrapi(c + 1, nj) : min(max(c + 1, 0), nj);  // the cell's right j-face
      const size_t row = size_t(row_cell(r + 1)) * (nj + 1);
      auto side = [&](int f) { return per_j ? -1 : (f == 0 ? 0 : (f == nj ? 1 : -1)); };
      face(S_JF, fj, nfj, row + cr, side(cr), row + cf, side(cf));
    }
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
