// Host check of the collision at a node's own scale (test infrastructure):
// collide_fx_at against collision_MRT with Guo's forcing by its moment matrix
// in long double, on states of many magnitudes of velocity and force, near
// equilibrium and at rest.  Prints per MRT rate set, velocity U and force F
//   mrt U F states declined ordinary ordinary_declined max_error
// with the error relative to the node's largest population before or after,
// and the ordinary states those whose force is below twice their largest
// population.
#include <cmath>
#include <cstdio>
#include <cstring>
#include <random>

#include "mrt_exact.cuh"

using namespace lbm;

int main() {
  for (int mrt = 1; mrt <= 3; ++mrt) {
    const Rates r = rate_set(mrt);
    const RatesT<double> rt = rates_t<double>(r);
    std::mt19937_64 rng(40 + mrt);
    std::normal_distribution<double> nd;
    for (double U : {0.0, 1e-11, 1e-9, 1e-7, 1e-5, 1e-3, 0.03})
      for (double ratio : {0.0, 1e-8, 1e-5, 1e-4, 1e-3, 1e-2, 0.1, 1.0, 10.0}) {
        const double Fa = (U > 0 ? U : 1e-5) * ratio;
        int declined = 0, states = 0, ordinary = 0, ordinary_declined = 0;
        double worst = 0.0;
        for (int it = 0; it < 300; ++it) {
          double v[3], F[3], f[19], u[3] = {0, 0, 0}, rho = 0;
          for (int a = 0; a < 3; ++a) { v[a] = U * nd(rng); F[a] = Fa * nd(rng); }
          const double rp = 3 * U * U * nd(rng);
          for (int q = 0; q < 19; ++q) {
            const double w = q == 0 ? 1. / 3 : (q <= 6 ? 1. / 18 : 1. / 36);
            const double cu = cix(q) * v[0] + ciy(q) * v[1] + ciz(q) * v[2];
            f[q] = w * (rp + 3 * cu + 4.5 * cu * cu - 1.5 * (v[0] * v[0] + v[1] * v[1] + v[2] * v[2]) +
                        0.02 * U * nd(rng));
            rho += f[q];
            u[0] += cix(q) * f[q];
            u[1] += ciy(q) * f[q];
            u[2] += ciz(q) * f[q];
          }
          for (int a = 0; a < 3; ++a) u[a] += 0.5 * F[a];
          Q o[19];
          exact(f, rho, u, F, r, o);
          double g[19], rho9 = rho;
          std::memcpy(g, f, sizeof f);
          ++states;
          double most = 0;
          for (int q = 0; q < 19; ++q) most = std::fmax(most, std::fabs(f[q]));
          const bool plain = std::fmax(std::fabs(F[0]), std::fmax(std::fabs(F[1]), std::fabs(F[2]))) < 2 * most;
          ordinary += plain;
          if (!collide_fx_at(g, false, rho9, u[0], u[1], u[2], F[0], F[1], F[2], rt)) {
            ++declined;
            ordinary_declined += plain;
            continue;
          }
          double big = 0, err = 0;
          for (int q = 0; q < 19; ++q) {
            big = std::fmax(big, std::fmax(std::fabs(f[q]), std::fabs((double)o[q])));
            err = std::fmax(err, std::fabs((double)(g[q] - o[q])));
          }
          if (big > 0) worst = std::fmax(worst, err / big);
        }
        std::printf("%d %g %g %d %d %d %d %.3e\n", mrt, U, Fa, states, declined, ordinary,
                    ordinary_declined, worst);
      }
  }
  return 0;
}
