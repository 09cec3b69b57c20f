// Host check of the integer collision core's roundings (test infrastructure):
// collide_fx_fixed_int, one step of stored fixed-point populations, against
// the moment matrix in long double on random near-equilibrium states.  Prints
// per MRT rate set and viscosity
//   mrt visc int_ok states declined mean rms xy_rms
// the mean and rms error of a population and the rms error of the stress
// sum c_x c_y f, in units of the storage, 2^-58; then, for collide_fx_at with
// the density summed, per rate set and velocity
//   mass mrt U states mean
// the mean of a node's mass error relative to its largest population.
#include <cmath>
#include <cstdio>
#include <random>

#include "mrt_exact.cuh"

using namespace lbm;

int main() {
  for (int mrt = 1; mrt <= 3; ++mrt)
    for (double visc : {0.0036, 3e-4, 1.2e-4, 1e-5, 1e-8}) {
      const Rates r = rate_set(mrt, visc);
      const RatesT<double> rt = rates_t<double>(r);
      std::mt19937_64 rng(9 + mrt);
      std::normal_distribution<double> nd;
      double sum = 0, s2 = 0, xy2 = 0;
      int declined = 0, states = 0;
      const Q unit = std::ldexp(Q(1), -kFxIn);
      for (int it = 0; it < 20000; ++it, ++states) {
        const double U = 0.04;
        double v[3];
        long long g[19], in[19], F[3], P[3];
        for (int a = 0; a < 3; ++a) {
          v[a] = U * nd(rng);
          F[a] = std::llround(std::ldexp(1e-5 * nd(rng), kFxF));
          P[a] = std::llround(std::ldexp(1e-5 * nd(rng), kFxF));
        }
        const double rp = 3 * U * U * nd(rng);
        for (int q = 0; q < 19; ++q) {
          const double w = q == 0 ? 1. / 3 : (q <= 6 ? 1. / 18 : 1. / 36);
          const double cu = cix(q) * v[0] + ciy(q) * v[1] + ciz(q) * v[2];
          const double f = w * (rp + 3 * cu + 4.5 * cu * cu -
                                1.5 * (v[0] * v[0] + v[1] * v[1] + v[2] * v[2]) + 0.02 * U * nd(rng));
          // (the low bits of a double this small are zero at 2^-58)
          g[q] = in[q] = (long long)std::ldexp(f, kFxIn) + (long long)(rng() & 15) - 8;
        }
        Q f[19], rho = 0, u[3] = {0, 0, 0}, force[3], o[19];
        for (int q = 0; q < 19; ++q) {
          f[q] = in[q] * unit;
          rho += f[q];
          u[0] += cix(q) * f[q];
          u[1] += ciy(q) * f[q];
          u[2] += ciz(q) * f[q];
        }
        for (int a = 0; a < 3; ++a) {
          force[a] = std::ldexp((Q)F[a], -kFxF);
          u[a] += std::ldexp((Q)P[a], -kFxF - 1);
        }
        exact(f, rho, u, force, r, o);
        if (!collide_fx_fixed_int(g, P[0], P[1], P[2], F[0], F[1], F[2], rt)) {
          ++declined;
          continue;
        }
        double xy = 0;
        for (int q = 0; q < 19; ++q) {
          const double e = (double)(g[q] - o[q] / unit);
          sum += e;
          s2 += e * e;
          xy += cix(q) * ciy(q) * e;
        }
        xy2 += xy * xy;
      }
      const double n = states - declined;
      std::printf("%d %g %d %d %d %.5f %.5f %.5f\n", mrt, visc, (int)rt.int_ok, states, declined,
                  sum / (19 * n), std::sqrt(s2 / (19 * n)), std::sqrt(xy2 / n));
    }
  for (int mrt = 1; mrt <= 3; ++mrt)
    for (double U : {1e-5, 0.01, 0.03}) {
      const RatesT<double> rt = rates_t<double>(rate_set(mrt));
      std::mt19937_64 rng(70 + mrt);
      std::normal_distribution<double> nd;
      double sum = 0;
      int states = 0;
      for (int it = 0; it < 20000; ++it) {
        double v[3], f[19], u[3] = {0, 0, 0}, rho = 0, big = 0;
        for (int a = 0; a < 3; ++a) v[a] = U * nd(rng);
        const double rp = 3 * U * U * nd(rng);
        Q mass = 0;
        for (int q = 0; q < 19; ++q) {
          const double w = q == 0 ? 1. / 3 : (q <= 6 ? 1. / 18 : 1. / 36);
          const double cu = cix(q) * v[0] + ciy(q) * v[1] + ciz(q) * v[2];
          f[q] = w * (rp + 3 * cu + 4.5 * cu * cu - 1.5 * (v[0] * v[0] + v[1] * v[1] + v[2] * v[2]) +
                      0.02 * U * nd(rng));
          u[0] += cix(q) * f[q];
          u[1] += ciy(q) * f[q];
          u[2] += ciz(q) * f[q];
          big = std::fmax(big, std::fabs(f[q]));
          mass -= f[q];
        }
        if (!collide_fx_at(f, true, rho, u[0], u[1], u[2], 0.0, 0.0, 0.0, rt)) continue;
        for (int q = 0; q < 19; ++q) mass += f[q];
        sum += (double)mass / big;
        ++states;
      }
      std::printf("mass %d %g %d %.3e\n", mrt, U, states, sum / states);
    }
  return 0;
}
