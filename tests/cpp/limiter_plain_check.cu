// The FP64 limiters of the stage kernels (minmod1, mc1, vanalbada1, vanleer1, limit4x2) against the
// plain expressions, written out here, over every pair of a set of values with zeros of both signs,
// subnormal, huge and infinite ones, NaN and random ones; on the host, and with the argument
// "device" on the GPU.
#include <cmath>
#include <cstdio>
#include <cstring>
#include <limits>
#include <random>
#include <vector>

#include "../../hyperboliconvergence_gb300/csrc/hc_physics.cuh"

using namespace hc;

static double plain(int kind, double a, double b) {
  const double tiny = std::numeric_limits<double>::min();
  switch (kind) {
    case LIM_MINMOD: return a > 0. ? std::fmin(a, std::fmax(b, 0.)) : std::fmax(a, std::fmin(b, 0.));
    case LIM_MC:
      return a > 0. ? std::fmax(0., std::fmin(0.5 * (a + b), std::fmin(2. * b, 2. * a)))
                    : std::fmin(0., std::fmax(0.5 * (a + b), std::fmax(2. * b, 2. * a)));
    case LIM_VANALBADA: return a * b < 0. ? 0. : (b * (a * a) + a * (b * b)) / (a * a + b * b + tiny);
    default: return (a * std::fabs(b) + std::fabs(a) * b) / (std::fabs(a) + std::fabs(b) + tiny);
  }
}
// smallest magnitude at which the plain quotients neither underflow nor overflow, and largest
static bool tame(double x) { return x == 0. || (std::fabs(x) > 1e-90 && std::fabs(x) < 1e90); }

constexpr int kKinds = 4;
__host__ __device__ inline int kind_of(int k) {
  return k == 0 ? LIM_MINMOD : k == 1 ? LIM_MC : k == 2 ? LIM_VANALBADA : LIM_VANLEER;
}
// limit() of a pair, and limit4x2's left and right sides with the pair's values
__host__ __device__ inline void evaluate(int kind, double a, double b, double* out) {
  const double a4[4] = {a, b, a, b}, l4[4] = {b, a, b, a}, r4[4] = {a, b, b, a};
  double l[4], r[4];
  limit4x2(kind, a4, l4, r4, l, r);
  out[0] = limit<double>(kind, a, b);
  out[1] = l[0]; out[2] = r[2]; out[3] = l[1]; out[4] = r[0];
}
__global__ void evaluate_all(const double* x, int n, double* out) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n * n) return;
  for (int k = 0; k < kKinds; ++k) evaluate(kind_of(k), x[i / n], x[i % n], out + (size_t(k) * n * n + i) * 5);
}

static int bad = 0;
static void check(const char* what, int kind, double a, double b, double got, double want) {
  bool ok = got == want || (std::isnan(got) && std::isnan(want));  // zeros compare equal whatever their sign
  if (kind == LIM_VANALBADA || kind == LIM_VANLEER) {
    if (tame(a) && tame(b)) {
      // the quotient's reciprocal is within 0.6 ulp, its other operations round five times on each side
      ok = ok || std::fabs(got - want) <= 6 * 2.3e-16 * std::fabs(want);
      // opposite signs: one of the two products that cancel is rounded, the other fused into the sum
      if (std::signbit(a) != std::signbit(b)) ok = ok || std::fabs(got) <= 1.2e-16 * std::fmin(std::fabs(a), std::fabs(b));
    } else {
      // where the plain products overflow or underflow: the slopes of opposite sign limit to 0, those
      // of one sign to no more than the larger (NaN and infinite arguments as the plain form has them)
      if (std::signbit(a) != std::signbit(b) && !std::isnan(a) && !std::isnan(b)) ok = ok || got == 0.;
      if (std::isfinite(a) && std::isfinite(b))
        ok = ok || !std::isfinite(want) || (std::isfinite(got) && std::fabs(got) <= 1.3 * std::fmax(std::fabs(a), std::fabs(b)));
    }
  }
  if (!ok && bad++ < 20) std::printf("%s kind %d a %.17g b %.17g: %.17g, plain %.17g\n", what, kind, a, b, got, want);
}

int main(int argc, char** argv) {
  const bool device = argc > 1 && !std::strcmp(argv[1], "device");
  const double inf = std::numeric_limits<double>::infinity(), nan = std::nan("");
  std::vector<double> x;
  for (double v : {0., 1., 1.5, 2., 3., 1. + 2.3e-16, 5e-324, 1e-310, 2.2250738585072014e-308, 1e-302, 1e-200, 1e-160, 1e-89,
                   1e89, 1e120, 1e154, 1e160, 1e301, 1.7976931348623157e308, inf, nan}) {
    x.push_back(v);
    x.push_back(-v);
  }
  std::mt19937_64 rng(17);
  std::uniform_real_distribution<double> u(-1., 1.), e(-40., 40.);
  for (int k = 0; k < 120; ++k) x.push_back(u(rng));
  for (int k = 0; k < 60; ++k) x.push_back(u(rng) * std::pow(10., e(rng)));
  const int n = int(x.size());
  std::vector<double> out(size_t(kKinds) * n * n * 5);
  if (device) {
    double *dx = nullptr, *dout = nullptr;
    if (cudaMalloc(&dx, n * 8) || cudaMalloc(&dout, out.size() * 8) || cudaMemcpy(dx, x.data(), n * 8, cudaMemcpyHostToDevice))
      return 2;
    evaluate_all<<<(n * n + 127) / 128, 128>>>(dx, n, dout);
    if (cudaMemcpy(out.data(), dout, out.size() * 8, cudaMemcpyDeviceToHost)) return 2;
  } else {
    for (int k = 0; k < kKinds; ++k)
      for (int i = 0; i < n * n; ++i) evaluate(kind_of(k), x[i / n], x[i % n], &out[(size_t(k) * n * n + i) * 5]);
  }
  for (int k = 0; k < kKinds; ++k)
    for (int i = 0; i < n * n; ++i) {
      const int kind = kind_of(k);
      const double a = x[i / n], b = x[i % n], *o = &out[(size_t(k) * n * n + i) * 5];
      check("limit", kind, a, b, o[0], plain(kind, a, b));
      check("left", kind, a, b, o[1], plain(kind, a, b));
      check("right", kind, a, b, o[2], plain(kind, a, b));
      check("left swapped", kind, b, a, o[3], plain(kind, b, a));
      check("right same", kind, a, a, o[4], plain(kind, a, a));
    }
  if (bad) std::printf("%d differ\n", bad);
  return bad ? 1 : 0;
}
