// collision_MRT with Guo's forcing by its moment matrix in long double, and the
// three MRT rate sets: what the host checks compare the kernels' forms with.
#pragma once
#include "lbm_collide.cuh"

typedef long double Q;

inline lbm::Rates rate_set(int m, double visc = 0.0036) {
  lbm::Rates r;
  const double s9 = 1.0 / (3 * visc + 0.5);
  r.s9 = r.s13 = s9;
  r.omegepsl = m == 1 ? 0.0 : 3.0;
  r.omegepslj = m == 1 ? -475.0 / 63.0 : -5.5;
  r.omegxx = m == 1 ? 0.0 : -0.5;
  if (m == 1) { r.s1 = 1.19; r.s2 = 1.4; r.s4 = 1.2; r.s10 = 1.4; r.s16 = 1.98; }
  else if (m == 3) { r.s1 = r.s2 = r.s10 = r.s16 = 1.8; r.s4 = s9; }
  else r.s1 = r.s2 = r.s4 = r.s10 = r.s16 = s9;
  return r;
}

template <typename V>
void exact(const V (&f)[19], Q rho, const V (&u)[3], const V (&F)[3], const lbm::Rates& r, Q (&o)[19]) {
  using lbm::cix;
  using lbm::ciy;
  using lbm::ciz;
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
