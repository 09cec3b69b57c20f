// Host check of the collision at a node's own scale (test infrastructure):
// collide_fx_at against collision_MRT with Guo's forcing by its moment matrix
// in long double, on states of many magnitudes of velocity and force, near
// equilibrium and at rest.  Prints per MRT rate set, velocity U and force F
//   mrt U F states declined ordinary ordinary_declined max_error
// with the error relative to the node's largest population before or after,
// and the ordinary states those whose force is below 1/128 of the velocity.
#include <cmath>
#include <cstdio>
#include <cstring>
#include <random>

#include "lbm_collide.cuh"

using namespace lbm;
typedef long double Q;

static Rates rate_set(int m) {
  Rates r;
  const double s9 = 1.0 / (3 * 0.0036 + 0.5);
  r.s9 = r.s13 = s9;
  r.omegepsl = m == 1 ? 0.0 : 3.0;
  r.omegepslj = m == 1 ? -475.0 / 63.0 : -5.5;
  r.omegxx = m == 1 ? 0.0 : -0.5;
  if (m == 1) { r.s1 = 1.19; r.s2 = 1.4; r.s4 = 1.2; r.s10 = 1.4; r.s16 = 1.98; }
  else if (m == 3) { r.s1 = r.s2 = r.s10 = r.s16 = 1.8; r.s4 = s9; }
  else r.s1 = r.s2 = r.s4 = r.s10 = r.s16 = s9;
  return r;
}

static void exact(const double (&f)[19], Q rho, const double (&u)[3], const double (&F)[3],
                  const Rates& r, Q (&o)[19]) {
  Q M[19][19], half[19], m[19], norm[19];
  const Q ux = u[0], uy = u[1], uz = u[2];
  for (int q = 0; q < 19; ++q) {
    const Q x = cix(q), y = ciy(q), z = ciz(q), s = x * x + y * y + z * z;
    const bool face = s == 1;
    const Q e = face ? -2 : 1, t = face ? -4 : 1;
    const Q row[19] = {1, s == 0 ? Q(-30) : (face ? Q(-11) : Q(8)),
                       s == 0 ? Q(12) : (face ? Q(-4) : Q(1)), x, t * x, y, t * y, z, t * z,
                       3 * x * x - s, e * (3 * x * x - s), y * y - z * z, e * (y * y - z * z),
                       x * y, y * z, x * z, x * (y * y - z * z), y * (z * z - x * x),
                       z * (x * x - y * y)};
    for (int k = 0; k < 19; ++k) M[k][q] = row[k];
    const Q w = q == 0 ? Q(1) / 3 : (q <= 6 ? Q(1) / 18 : Q(1) / 36);
    const Q cu = x * ux + y * uy + z * uz, cF = x * F[0] + y * F[1] + z * F[2];
    const Q uF = ux * F[0] + uy * F[1] + uz * F[2];
    half[q] = w * (3 * cF + 9 * cF * cu - 3 * uF) / 2;
  }
  for (int k = 0; k < 19; ++k) {
    m[k] = norm[k] = 0;
    for (int q = 0; q < 19; ++q) {
      m[k] += M[k][q] * (f[q] + half[q]);
      norm[k] += M[k][q] * M[k][q];
    }
  }
  const Q t = ux * ux + uy * uy + uz * uz, e6 = 2 * ux * ux - uy * uy - uz * uz, e8 = uy * uy - uz * uz;
  const Q eq[19] = {0, -11 * rho + 19 * t, r.omegepsl * rho + r.omegepslj * t, 0, -2 * ux / 3, 0,
                    -2 * uy / 3, 0, -2 * uz / 3, e6, r.omegxx * e6, e8, r.omegxx * e8,
                    ux * uy, uy * uz, ux * uz, 0, 0, 0};
  const double rate[19] = {0, r.s1, r.s2, 0, r.s4, 0, r.s4, 0, r.s4, r.s9, r.s10, r.s9, r.s10,
                           r.s13, r.s13, r.s13, r.s16, r.s16, r.s16};
  for (int k = 0; k < 19; ++k) m[k] -= rate[k] * (m[k] - eq[k]);
  m[0] = rho;
  m[3] = ux;
  m[5] = uy;
  m[7] = uz;
  for (int q = 0; q < 19; ++q) {
    o[q] = half[q];
    for (int k = 0; k < 19; ++k) o[q] += M[k][q] * m[k] / norm[k];
  }
}

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
          auto largest = [](const double (&a)[3]) {
            return std::fmax(std::fabs(a[0]), std::fmax(std::fabs(a[1]), std::fabs(a[2])));
          };
          const bool plain = 128 * largest(F) < largest(u);
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
