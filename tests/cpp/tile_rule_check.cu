// The FP64 tile by the mesh's size (f64_auto_tile): every mesh that 16 x 16 tiles can be launched on
// gets a shape whose launch is within the grid's limits, and small meshes keep the small tiles.  The
// rows of an FP32 strip run (strip_run_rows): no mesh gets more work items than it may have.
// Host code: no GPU.
#include <cstdio>

#include "../../hyperboliconvergence_gb300/csrc/hc_launch.h"

using namespace hc;

int main() {
  int bad = 0;
  auto rows = [](int tile, int ni) { return tile == TILE_8x8 ? (ni + 7) / 8 : tile == TILE_4x8 ? (ni + 3) / 4 : (ni + 15) / 16; };
  const int nis[] = {3, 40, 128, 300, 512, 4096, 100000, 262140, 262141, 300000, 524280, 524281, 600000, 1000000, 1048560};
  const int njs[] = {3, 8, 17, 24, 40, 128, 200};
  for (int sms : {1, 148, 152, 160})
    for (int ni : nis)
      for (int nj : njs) {
        if ((long long)(ni + 1) * (nj + 1) > (1ll << 28)) continue;
        const int t = f64_auto_tile(ni, nj, sms);
        if (rows(t, ni) > 65535) {
          std::printf("%d x %d, %d SMs: tile %d has %d rows of tiles\n", ni, nj, sms, t, rows(t, ni));
          ++bad;
        }
      }
  if (f64_auto_tile(40, 40, 152) != TILE_4x8 || f64_auto_tile(512, 1024, 152) != TILE_16x16_H) ++bad;
  for (int sms : {1, 152})
    for (int ni : nis)
      for (int nj : {3, 28, 29, 4000, 100000, 1834980, 1834981, 1900000}) {
        if ((long long)(ni + 1) * (nj + 1) > (1ll << 28)) continue;
        const bool can = (long long)strip_count(nj) * strip_runs(ni, 64) <= 0xffff;
        const int rows = strip_run_rows(1, [&](int) { return ni; }, [&](int) { return nj; }, sms, 0xffff);
        const int any = strip_run_rows(1, [&](int) { return ni; }, [&](int) { return nj; }, sms);
        if ((rows > 0) != can || (rows > 0 && (long long)strip_count(nj) * strip_runs(ni, rows) > 0xffff) || any < 1) {
          std::printf("strips of %d x %d, %d SMs: %d rows, %d without a limit\n", ni, nj, sms, rows, any);
          ++bad;
        }
      }
  return bad ? 1 : 0;
}
