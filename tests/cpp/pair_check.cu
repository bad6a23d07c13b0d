// Packed pairs of double-float values against the scalar operations of hc_df64.cuh, both on the
// device (every operation must give the same bits), and the split of a double by its bits
// against the split by conversions.  Prints the number of mismatches of each.
#include "../../hyperboliconvergence_gb300/csrc/hc_pair.cuh"

#include <cmath>
#include <cstdio>
#include <random>
#include <vector>

using namespace hc;

__device__ bool same(float a, float b) { return a == b || (a != a && b != b); }
__device__ bool same(df64 a, df64 b) { return same(a.hi, b.hi) && same(a.lo, b.lo); }

enum { ADD, SUB, MUL, DIV, RCP, ALBADA, LEER, MINMOD, STATE, SPLIT, ROE, OPS };

__global__ void check(const double* x, int n, int* bad) {
  const int k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= n) return;
  auto at = [&](int o) { return x[(k + o * 7919) % n]; };
  const df64 a = dd::split(at(0)), b = dd::split(at(1)), c = dd::split(at(2)), d = dd::split(at(3));
  const df2 p = pair(a, b), q = pair(c, d);
  auto note = [&](int op, df2 r, df64 l, df64 h) {
    if (!same(lo(r), l) || !same(hi(r), h)) atomicAdd(&bad[op], 1);
  };
  note(ADD, p + q, a + c, b + d);
  note(SUB, p - q, a - c, b - d);
  note(MUL, p * q, a * c, b * d);
  note(DIV, p / q, a / c, b / d);
  note(RCP, rcp(p), dd::rcp(a), dd::rcp(b));
  note(ALBADA, limit2(LIM_VANALBADA, d, p), limit<df64>(LIM_VANALBADA, d, a), limit<df64>(LIM_VANALBADA, d, b));
  note(LEER, limit2(LIM_VANLEER, d, p), limit<df64>(LIM_VANLEER, d, a), limit<df64>(LIM_VANLEER, d, b));
  note(MINMOD, limit2(LIM_MINMOD, d, p), limit<df64>(LIM_MINMOD, d, a), limit<df64>(LIM_MINMOD, d, b));
  Gas<df64> g{};
  g.gamma = df64(1.4); g.gamma1 = df64(2.5);
  const df2 s[4] = {p, q, pair(fabs(c), fabs(a)), pair(fabs(d), fabs(b))};
  const StPair sp = prim_states(g, s);
  const St<df64> l = left_state(sp), r = right_state(sp);
  const St<df64> l0 = prim_state_ir(g, a, c, fabs(c), fabs(d), dd::rcp(fabs(c)));
  const St<df64> r0 = prim_state_ir(g, b, d, fabs(a), fabs(b), dd::rcp(fabs(a)));
  if (!same(l.h, l0.h) || !same(r.h, r0.h) || !same(l.a2, l0.a2) || !same(r.u2, r0.u2)) atomicAdd(&bad[STATE], 1);
  // a flow: velocities of some units about a density and a pressure near 1, so that the averaged
  // sound speed is real; sub-, trans- and supersonic faces
  g.gm1 = df64(0.4);
  const df64 sc(float(1.0 / 1024.0), 0.f);
  const df2 t[4] = {p * pair(sc), q * pair(sc), pair(df64(1.0)) + pair(fabs(a), fabs(c)) * pair(sc),
                    pair(df64(1.0)) + pair(fabs(b), fabs(d)) * pair(sc)};
  const StPair f = prim_states(g, t);
  const df64 nx = df64(0.6), ny = df64(-0.8), A = df64(1.75);
  for (int want = 0; want < 2; ++want) {
    const Flux5<df64> m = roe_flux_pairs<false>(g, nx, ny, A, f, want), w = roe_flux_pairs<true>(g, nx, ny, A, f, want);
    const Flux5<df64> m0 = roe_flux<df64, false>(g, nx, ny, A, left_state(f), right_state(f), want);
    const Flux5<df64> w0 = roe_flux<df64, true>(g, nx, ny, A, left_state(f), right_state(f), want);
    bool ok = same(m.lam, m0.lam) && same(w.lam, w0.lam);
    for (int v = 0; v < 4; ++v) ok = ok && same(m.f[v], m0.f[v]) && same(w.f[v], w0.f[v]) && m.f[v].hi == m.f[v].hi;
    if (!ok) atomicAdd(&bad[ROE], 1);
  }
  if (!same(dd::split(at(0)), df64(at(0)))) atomicAdd(&bad[SPLIT], 1);
}

int main() {
  std::mt19937_64 g(5);
  std::uniform_real_distribution<double> u(-1.0, 1.0);
  std::vector<double> x;
  // the magnitudes of the products and squares stay inside FP32's range
  for (int k = 0; k < 1 << 18; ++k) x.push_back(u(g) * std::ldexp(1.0, int(g() % 21) - 10));
  for (double e : {1.0, 0.5, 4096.0, 1e-3}) {
    const float f = float(e);
    const double ulp = std::nextafterf(f, 2 * f) - f;
    // ties and their neighbours, carries into the exponent, values with a zero second part
    for (double v : {double(f), f + 0.5 * ulp, f + 1.5 * ulp, f - 0.25 * ulp, f + 0.5 * ulp * (1 + 1e-8),
                     f + 0.5 * ulp * (1 - 1e-8), 2 * f - 0.25 * ulp, 2.0 * f - 1e-16 * f})
      for (double sgn : {1.0, -1.0}) x.push_back(sgn * v);
  }
  const size_t plain = x.size();
  std::vector<double> wide = x;
  for (int k = 0; k < 1 << 16; ++k) wide.push_back(u(g) * std::ldexp(1.0, int(g() % 300) - 170));
  for (double v : {0.0, -0.0, 1e-310, 3.4e38, 1e39, 1e300, double(INFINITY), -double(INFINITY), double(NAN)}) wide.push_back(v);
  int bad[2][OPS] = {};
  double* d;
  int* b;
  if (cudaMalloc(&d, wide.size() * 8) != cudaSuccess || cudaMalloc(&b, sizeof(bad)) != cudaSuccess) return 2;
  cudaMemset(b, 0, sizeof(bad));
  cudaMemcpy(d, x.data(), plain * 8, cudaMemcpyHostToDevice);
  check<<<unsigned((plain + 255) / 256), 256>>>(d, int(plain), b);
  cudaMemcpy(d, wide.data(), wide.size() * 8, cudaMemcpyHostToDevice);
  check<<<unsigned((wide.size() + 255) / 256), 256>>>(d, int(wide.size()), b + OPS);
  if (cudaMemcpy(bad, b, sizeof(bad), cudaMemcpyDeviceToHost) != cudaSuccess) return 2;
  static const char* names[OPS] = {"add", "sub", "mul", "div", "rcp", "vanalbada", "vanleer", "minmod", "state", "split", "roe"};
  for (int o = 0; o < OPS; ++o) std::printf("%s %d\n", names[o], bad[0][o]);
  std::printf("split_wide %d\n", bad[1][SPLIT]);
  return 0;
}
