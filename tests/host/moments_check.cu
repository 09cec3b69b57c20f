// Host check of the integer density and momentum sums (test infrastructure):
// fx_moments against long double, at magnitudes up to the ends of FP64's range.
// Prints per magnitude
//   magnitude states taken non_finite_missed max_error
// the error relative to the sum of the magnitudes, and the states taken whose
// exact sums are beyond FP64's range but whose result is not infinite.
#include <cmath>
#include <cstdio>
#include <random>

#include "mrt_exact.cuh"

using namespace lbm;

int main() {
  std::mt19937_64 rng(5);
  std::uniform_real_distribution<double> ud(-1.0, 1.0);
  for (double magnitude : {1e-300, 1e-200, 1e-30, 1e-3, 1.0, 1e30, 1e300, 1e306, 1e307, 3e307, 1e308, 1.7e308}) {
    int taken = 0, missed = 0;
    double worst = 0;
    for (int it = 0; it < 2000; ++it) {
      double f[19], got[4];
      Q sum[4] = {0, 0, 0, 0}, all = 0;
      for (int q = 0; q < 19; ++q) {
        // (every other state of one sign: sums beyond the range)
        f[q] = magnitude * (it & 1 ? std::fabs(ud(rng)) : ud(rng));
        const int c[4] = {1, cix(q), ciy(q), ciz(q)};
        for (int k = 0; k < 4; ++k) sum[k] += c[k] * (Q)f[q];
        all += std::fabs((Q)f[q]);
      }
      if (!fx_moments(f, got[0], got[1], got[2], got[3])) continue;
      ++taken;
      for (int k = 0; k < 4; ++k) {
        if (std::isinf((double)sum[k])) missed += !std::isinf(got[k]);
        else worst = std::fmax(worst, (double)(std::fabs(got[k] - sum[k]) / all));
      }
    }
    std::printf("%g %d %d %d %.3e\n", magnitude, 2000, taken, missed, worst);
  }
  return 0;
}
