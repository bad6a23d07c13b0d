// The isentropic powers of the far fields (pow_gas): within the type's rounding of the power of the
// exponent that is given, also where it lies close to a half integer without being one.  Host code:
// no GPU.
#include <cmath>
#include <cstdio>

#include "../../hyperboliconvergence_gb300/csrc/hc_physics.cuh"

using namespace hc;

static int bad = 0;
// gas: the exponents 1/(gamma - 1) as make_gas forms them, in which gamma's own rounding (half an ulp
// of gamma, over gamma - 1) is no information
template <class R> static void check(double gamma, double eps, bool gas) {
  const R e = make_gas<R>(gamma, 287.058, 0.3).gamma1;
  for (double x : {1e-4, 0.02, 0.3, 0.77, 0.999, 1.0, 1.0001, 1.3, 2.9, 40.0, 1e4}) {
    const R xr = R(x);
    if (std::fabs(double(e) * std::log10(x)) > (sizeof(R) == 4 ? 37 : 300)) continue;  // beyond the type
    const long double want = powl((long double)xr, (long double)e), got = pow_gas(xr, e);
    // up to nine products and a root; and e's own uncertainty where the exponent is a gas's
    const long double tol = 10 * 0.5L * eps + (gas ? (long double)e * e * 1.2e-16L * fabsl(logl((long double)xr)) * 1.5L : 0.0L);
    if (!(fabsl(got - want) <= tol * want)) {
      if (bad++ < 10)
        std::printf("gamma %.17g e %.17g x %g: %.17Lg, power %.17Lg, relative %.3Lg\n", gamma, double(e), x, got, want,
                    (got - want) / want);
    }
  }
}

int main() {
  for (double gamma : {1.4, 5. / 3., 1.2, 9. / 7., 1.5, 2., 3., 1.25, 4. / 3., 1.3, 1.66, 1.667, 1.405, 1.1}) {
    check<double>(gamma, 2.3e-16, true);
    check<float>(gamma, 1.2e-7, true);
    // gammas near it
    for (double d : {1e-14, 3e-13, 1e-10, 1e-8, 6e-8, 1.2e-7, 3e-7, 1e-6, 1e-5, -1e-14, -1e-10, -1e-8, -1e-7, -1e-6}) {
      check<double>(gamma + d, 2.3e-16, true);
      check<float>(gamma + d, 1.2e-7, true);
    }
  }
  return bad ? 1 : 0;
}
