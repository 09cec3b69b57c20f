// Host check of the nearest-image sweeps (test infrastructure): sweep_fast
// against sweep_events, the reference's expressions, for centres over and
// around the box, at and around the ties, and for the end states of earlier
// sweeps.  Prints "n taken_share mismatches cases" per box length.
#include <cmath>
#include <cstdio>
#include <random>

#include "lbm_sweeps.cuh"

using namespace lbm;

static bool same(double a, double b) { return std::memcmp(&a, &b, sizeof a) == 0; }

int main() {
  std::mt19937_64 rng(11);
  for (int n : {4, 5, 7, 32, 33, 95, 130, 256, 1001}) {
    const int nh = n / 2;
    std::uniform_real_distribution<double> in_box(0.0, n), wide(-1.5 * n, 2.5 * n);
    long long taken = 0, bad = 0, cases = 0;
    auto one = [&](double c0) {
      double c = c0;
      for (int s = 0; s < 4; ++s) {
        const SweepEv e = sweep_events(c, n, nh);
        SweepEv f;
        double cf = c;
        ++cases;
        if (sweep_fast(cf, n, nh, &f)) {
          ++taken;
          bool ok = f.nev == e.nev && f.ok == e.ok && same(f.v0, e.v0) && same(cf, sweep_value(e, n));
          for (int k = 0; ok && k < e.nev; ++k) ok = f.j[k] == e.j[k] && same(f.v[k], e.v[k]);
          bad += !ok;
        } else {
          bad += !same(cf, c);
        }
        c = sweep_value(e, n);
      }
    };
    for (int i = 0; i < 20000; ++i) one(in_box(rng));
    for (int i = 0; i < 5000; ++i) one(wide(rng));
    // ties: n/2 + 1/2, half-integers, integers, 0 and n, an ulp to either side and a little more
    for (int k = -2; k <= 2 * n + 2; ++k)
      for (double d : {0.0, 1e-15, 1e-13, 1e-11, 1e-9, 1e-6})
        for (double sg : {-1.0, 1.0}) {
          const double b = 0.5 * k;
          one(b + sg * d * (1.0 + std::fabs(b)));
          one(std::nextafter(b, sg * 1e9));
        }
    for (double v : {1e300, -1e300, 4194304.0, std::nan(""), (double)INFINITY}) {
      double c = v;
      SweepEv f;
      ++cases;
      bad += sweep_fast(c, n, nh, &f);
    }
    std::printf("%d %.4f %lld %lld\n", n, (double)taken / cases, bad, cases);
  }
  return 0;
}
