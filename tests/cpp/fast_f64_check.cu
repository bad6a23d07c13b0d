// Device check of the FP64 reciprocal, quotient and square roots of the stage arithmetic and of
// the bitwise limiters, clamps and comparisons (hc_physics.cuh).  Relative errors against long
// double must stay below the bounds of their derivation (the step's truncation, below 2^-57,
// plus the roundings): 2^-52 for 1/x and the square roots, 2^-51.5 for the quotient.  Outside
// the window, and for the selections, the device must give the host's plain expression.
#include "../../hyperboliconvergence_gb300/csrc/hc_physics.cuh"

#include <cmath>
#include <cstdio>
#include <cstring>
#include <random>
#include <vector>

using namespace hc;

namespace {
constexpr int NOUT = 11;

__global__ void eval(const double* x, const double* y, double* o, int n) {
  const int k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= n) return;
  double* p = o + size_t(NOUT) * k;
  p[0] = rcp_fast(x[k]);
  p[1] = div_fast(y[k], x[k]);
  sqrt_rcp(x[k], p[2], p[3]);
  sqrt_fast(x[k], p[4]);
  p[5] = clamp01(x[k]);
  p[6] = abs_above_one(x[k]) ? 1.0 : 0.0;
  p[7] = max_pos(fabs(x[k]), fabs(y[k]));
  const double a[4] = {x[k], x[k], y[k], -x[k]}, b[4] = {y[k], -y[k], x[k], x[k] * 0.75};
  double l[4], r[4];
  const int kinds[3] = {LIM_VANALBADA, LIM_VANLEER, LIM_MINMOD};
  for (int m = 0; m < 3; ++m) {
    limit4x2(kinds[m], a, b, b, l, r);
    double worst = 0;
    for (int v = 0; v < 4; ++v) {
      const double want = limit<double>(kinds[m], a[v], b[v]);
      const double s = fmin(fabs(a[v]), fabs(b[v]));  // every one of these slopes is of this size at most
      double e = (l[v] == want || (isnan(l[v]) && isnan(want))) ? 0.0 : fabs(l[v] - want) / fmax(2 * s, 1e-300);
      if (!(l[v] == r[v] || (isnan(l[v]) && isnan(r[v])))) e = 1.0;
      if (!(e <= 1.0)) e = 1.0;
      worst = fmax(worst, e);
    }
    p[8 + m] = worst;
  }
}

bool same(double a, double b) { return a == b || (std::isnan(a) && std::isnan(b)); }
int bad = 0;
void rel(const char* what, double got, long double want, double bound, double x, double y) {
  const long double e = fabsl((long double)got - want) / fabsl(want);
  if (!(e <= bound) && bad++ < 20) std::printf("%s(%g, %g): %.17g, off by %.3Lg > %.3g\n", what, x, y, got, e, bound);
}
}  // namespace

int main() {
  std::vector<double> x, y;
  std::mt19937_64 rng(7);
  std::uniform_real_distribution<double> m(1.0, 2.0);
  std::uniform_int_distribution<int> e(-330, 330), near0(-3, 3);
  for (int k = 0; k < 40000; ++k) {
    x.push_back(std::ldexp(m(rng), k % 2 ? e(rng) : near0(rng)) * (k % 5 ? 1 : -1));
    y.push_back(std::ldexp(m(rng), k % 2 ? e(rng) : near0(rng)));
  }
  const double edge[] = {0.0, -0.0, 4.9e-324, 2.3e-308, std::ldexp(1.0, -1000), std::ldexp(1.0, -1001), 1.0, -1.0,
                         std::nextafter(1.0, 0.0), std::nextafter(1.0, 2.0), std::ldexp(1.0, 999), std::ldexp(1.9, 999),
                         std::ldexp(1.0, 1000), 1.7e308, INFINITY, -INFINITY, NAN};
  for (double a : edge)
    for (double b : edge) { x.push_back(a); y.push_back(b); }
  const int n = int(x.size());
  double *dx, *dy, *dout;
  std::vector<double> o(size_t(NOUT) * n);
  if (cudaMalloc(&dx, n * 8) || cudaMalloc(&dy, n * 8) || cudaMalloc(&dout, o.size() * 8)) return 2;
  cudaMemcpy(dx, x.data(), n * 8, cudaMemcpyHostToDevice);
  cudaMemcpy(dy, y.data(), n * 8, cudaMemcpyHostToDevice);
  eval<<<(n + 255) / 256, 256>>>(dx, dy, dout, n);
  if (cudaMemcpy(o.data(), dout, o.size() * 8, cudaMemcpyDeviceToHost) != cudaSuccess) return 2;
  const double ulp = std::ldexp(1.0, -52);
  for (int k = 0; k < n; ++k) {
    const double a = x[k], b = y[k], *p = &o[size_t(NOUT) * k];
    const bool normal = std::isnormal(a) && std::isnormal(1.0 / a), pos = normal && a > 0;
    if (normal) rel("rcp", p[0], 1.0L / a, ulp, a, b);
    else if (!same(p[0], 1.0 / a) && bad++ < 20) std::printf("rcp(%g): %g\n", a, p[0]);
    const double q = b / a;
    if (normal && std::isnormal(b) && std::isnormal(q)) rel("div", p[1], (long double)b / a, 1.42 * ulp, a, b);
    else if (!normal && !same(p[1], q) && bad++ < 20) std::printf("div(%g, %g): %g\n", b, a, p[1]);
    if (pos) {
      rel("sqrt", p[2], sqrtl(a), ulp, a, b);
      rel("rsqrt", p[3], 1.0L / sqrtl(a), ulp, a, b);
      rel("sqrt", p[4], sqrtl(a), ulp, a, b);
    } else if ((!same(p[2], std::sqrt(a)) || !same(p[3], 1.0 / std::sqrt(a)) || !same(p[4], std::sqrt(a))) && bad++ < 20) {
      std::printf("sqrt(%g): %g %g %g\n", a, p[2], p[3], p[4]);
    }
    if (!same(p[5], std::fmin(std::fmax(a, 0.0), 1.0)) && bad++ < 20) std::printf("clamp01(%g): %g\n", a, p[5]);
    if (p[6] != (std::fabs(a) > 1.0 ? 1.0 : 0.0) && bad++ < 20) std::printf("abs_above_one(%g)\n", a);
    if (!same(p[7], std::fmax(std::fabs(a), std::fabs(b))) && bad++ < 20) std::printf("max_pos(%g, %g): %g\n", a, b, p[7]);
    // the limiters where neither expression over- or underflows
    if (std::isfinite(a) && std::isfinite(b) && std::fabs(a) < 1e100 && std::fabs(b) < 1e100 && std::fabs(a) > 1e-100 &&
        std::fabs(b) > 1e-100)
      for (int v = 8; v < 11; ++v)
        if (!(p[v] <= 8 * ulp) && bad++ < 20) std::printf("limiter %d (%g, %g): off by %g\n", v - 8, a, b, p[v]);
  }
  std::printf("%d values, %d bad\n", n, bad);
  return bad ? 1 : 0;
}
