// Bessel function K0 in double precision.
#pragma once
#include <cmath>

namespace msx {

// K0(x) = int_0^inf exp(-x cosh u) du (x > 0).  The integrand is analytic and
// decays double-exponentially in the strip |Im u| < pi/2, so the trapezoidal
// rule with step h converges like exp(-pi^2 / h) while the peak at u = 0, of
// width 1/sqrt(x), is wide against h.  The relative error of h = 1/4 is 1e-17 at
// x = 2, 1.1e-16 at 3, 6e-16 at 4 and 5e-15 at 6: it serves x < 3, where it is
// lost in the rounding (6.3e-16 at most over [0.1, 3]; h = 1/8, which takes twice
// the terms, 7.2e-16 over [0.1, 8]), and h = 1/8 the larger x.  The sum stops once a
// term falls below 1e-18 of the running sum: cosh(u) < 1 + 42 / x, so u < 7 for every
// x >= 0.1.
constexpr int kCoshTable = 64;  // cosh(k / 8)
struct CoshTable {
  double v[kCoshTable];
  constexpr CoshTable() : v() {
    for (int k = 0; k < kCoshTable; ++k) {
      const double x = k / 8.0;
      double term = 1.0, sum = 1.0;  // all terms positive: x < 8 needs 30 of them
      for (int n = 1; n < 40; ++n) {
        term *= x * x / double((2 * n - 1) * (2 * n));
        sum += term;
      }
      v[k] = sum;
    }
  }
};

__host__ __device__ inline double bessel_k0(double x, const double* cosh8) {
  const int step = x < 3.0 ? 2 : 1;  // in units of 1/8
  double sum = 0.5 * exp(-x);
  for (int k = step; k < kCoshTable; k += step) {
    const double term = exp(-x * cosh8[k]);
    sum += term;
    if (term < 1e-18 * sum) break;
  }
  return 0.125 * step * sum;
}

}  // namespace msx
