// The FP32 square root of the stage kernels: within an ulp of the root over every exponent, infinity,
// NaN, zero and negative arguments as the library's root has them.
#include <cmath>
#include <cstdio>
#include <cstring>
#include <limits>
#include <vector>

#include "../../hyperboliconvergence_gb300/csrc/hc_physics.cuh"

using namespace hc;

__global__ void roots(const float* x, int n, float* s, float* s2, float* r) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  sqrt_fast(x[i], s[i]);
  sqrt_rcp(x[i], s2[i], r[i]);
}

int main() {
  const float inf = std::numeric_limits<float>::infinity();
  std::vector<float> x = {0.f, -0.f, inf, -inf, NAN, -1.f, -1e30f, -FLT_MIN, FLT_MIN, FLT_MAX, 1.f, 4.f, 2.f};
  for (int e = -126; e <= 127; ++e)
    for (int k = 0; k < 64; ++k) x.push_back(std::ldexp(1.f + float(k) / 64.f + float(k * k % 97) * 1.2e-7f, e));
  const int n = int(x.size());
  float *dx, *ds, *d2, *dr;
  if (cudaMalloc(&dx, n * 4) || cudaMalloc(&ds, n * 4) || cudaMalloc(&d2, n * 4) || cudaMalloc(&dr, n * 4) ||
      cudaMemcpy(dx, x.data(), n * 4, cudaMemcpyHostToDevice))
    return 2;
  roots<<<(n + 127) / 128, 128>>>(dx, n, ds, d2, dr);
  std::vector<float> s(n), s2(n);
  if (cudaMemcpy(s.data(), ds, n * 4, cudaMemcpyDeviceToHost) || cudaMemcpy(s2.data(), d2, n * 4, cudaMemcpyDeviceToHost)) return 2;
  int bad = 0;
  for (int i = 0; i < n; ++i) {
    const float want = std::sqrt(x[i]);
    const float ulp = std::nextafter(want, inf) - want;
    const bool ok = std::isnan(want) ? std::isnan(s[i]) : (s[i] == want || std::fabs(s[i] - want) <= ulp);
    if ((!ok || std::memcmp(&s[i], &s2[i], 4)) && !(std::isnan(s[i]) && std::isnan(s2[i]) && ok) && bad++ < 10)
      std::printf("sqrt(%g): %g %g, root %g\n", x[i], s[i], s2[i], want);
  }
  return bad ? 1 : 0;
}
