// The bounded wait of the strip kernel's record ring (hc_stage_warp.cuh) with every other warp of a
// block meeting a copy that falls 16 bytes short of what its barrier expects.
#include <cstdio>
#include <vector>

#include "../../hyperboliconvergence_gb300/csrc/hc_stage_warp.cuh"

using namespace hc;

constexpr int kRows = 7, kShort = 3;  // rows a warp fetches, the one that stays short
struct Lane {
  int dead, good;        // the lane's ring after the march, rows whose values were right
  unsigned used, read;
};

__global__ void ring_kernel(const float* rows, StepInfo* info, Lane* out) {
  extern __shared__ __align__(128) unsigned char smem[];
  StripRing ring = strip_ring(smem, true);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const bool shorted = warp % 2 == 1;
  int good = 0;
  for (int r = 0; r < kStripSlots; ++r) strip_fetch(ring, rows + r * kStripRow, kStripRow, lane, shorted && r == kShort);
  for (int r = 0; r < kRows; ++r) {
    const float* s = strip_wait(ring, info + warp);
    bool ok = true;
    for (int k = lane; k < kStripRow; k += 32) ok = ok && s[k] == rows[r * kStripRow + k];
    good += ok;
    // every lane is here: a warp whose lanes had parted would hang or mix these up
    if (__shfl_sync(0xffffffffu, r, (lane + 1) & 31) != r) good = -100;
    __syncwarp();
    if (r + kStripSlots < kRows)
      strip_fetch(ring, rows + (r + kStripSlots) * kStripRow, kStripRow, lane, shorted && r + kStripSlots == kShort);
  }
  out[threadIdx.x] = {ring.dead ? 1 : 0, good, ring.used, ring.read};
}

int main() {
  std::vector<float> h(size_t(kRows) * kStripRow);
  for (size_t k = 0; k < h.size(); ++k) h[k] = float(k % 100003);
  float* rows = nullptr;
  StepInfo* info = nullptr;
  Lane* out = nullptr;
  constexpr int kThreads = 32 * kStripWarps;
  if (cudaMalloc(&rows, h.size() * 4) || cudaMalloc(&info, kStripWarps * sizeof(StepInfo)) ||
      cudaMalloc(&out, kThreads * sizeof(Lane)) || cudaMemset(info, 0, kStripWarps * sizeof(StepInfo)) ||
      cudaMemcpy(rows, h.data(), h.size() * 4, cudaMemcpyHostToDevice))
    return 2;
  ring_kernel<<<1, kThreads, kStripSmem>>>(rows, info, out);
  std::vector<Lane> lanes(kThreads);
  std::vector<StepInfo> st(kStripWarps);
  if (cudaMemcpy(lanes.data(), out, kThreads * sizeof(Lane), cudaMemcpyDeviceToHost) ||
      cudaMemcpy(st.data(), info, kStripWarps * sizeof(StepInfo), cudaMemcpyDeviceToHost)) {
    std::printf("%s\n", cudaGetErrorString(cudaGetLastError()));
    return 2;
  }
  int bad = 0;
  for (int t = 0; t < kThreads; ++t) {
    const bool shorted = (t / 32) % 2 == 1;
    // a warp dies as a whole at the short row, whose rows before were right, and stays there, having
    // waited for what it had fetched; the others read all
    const bool ok = shorted ? lanes[t].dead == 1 && lanes[t].good >= kShort && lanes[t].read == kShort &&
                                  lanes[t].used == kShort + kStripSlots
                            : lanes[t].dead == 0 && lanes[t].good == kRows && lanes[t].read == kRows &&
                                  lanes[t].used == kRows;
    if (!ok) {
      std::printf("thread %d: dead %d good %d used %u read %u\n", t, lanes[t].dead, lanes[t].good, lanes[t].used, lanes[t].read);
      ++bad;
    }
  }
  for (int w = 0; w < kStripWarps; ++w)
    if (st[w].status != (w % 2 == 1 ? ST_TIMEOUT : ST_OK)) {
      std::printf("warp %d: status %d\n", w, st[w].status);
      ++bad;
    }
  return bad ? 1 : 0;
}
