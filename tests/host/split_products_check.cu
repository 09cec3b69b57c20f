// Host check of the integer collision core's products (test infrastructure).
// dot_shift (sums of 64-bit products by signed 32-bit halves, one rounding)
// against the exact 128-bit sum, at the edges of its operands and at random;
// split against its operand; and the factors of rates_t at the rate sets'
// limits.  Prints
//   split bad count
//   dot S n max_error   (units of the result; 1/2 + n/4 * 2^(64-S) allowed)
//   rates int_ok(1) int_ok(2) int_ok(3) int_ok(s9 = 2)
#include <cmath>
#include <cstdio>
#include <random>

#include "lbm_collide.cuh"

using namespace lbm;

static long long bad_split = 0, n_split = 0;
static Split checked(long long v) {
  const Split s = split(v);
  ++n_split;
  bad_split += ((__int128)s.h * ((__int128)1 << 32) + s.l) != (__int128)v;
  return s;
}

template <int S, int n>
void dots(std::mt19937_64& rng) {
  const long long edge[] = {0, 1, -1, 0x7fffffffLL, 0x80000000LL, -0x80000000LL, 0x80000001LL,
                            0xffffffffLL, 1LL << 32, -(1LL << 32), (1LL << 58) - 1, -(1LL << 58)};
  const int ne = sizeof edge / sizeof edge[0];
  double worst = 0.0;
  for (int it = 0; it < 400000; ++it) {
    Split a[n], b[n];
    __int128 exact = 0;
    for (int i = 0; i < n; ++i) {
      // |a| < 2^60, |b| < 2^61: the sums of middle terms stay below 2^63
      const long long x = it < ne * ne ? edge[it % ne] : (long long)rng() >> (4 + rng() % 40);
      const long long y = it < ne * ne ? edge[it / ne] : (long long)rng() >> (3 + rng() % 40);
      a[i] = checked(x);
      b[i] = checked(y);
      exact += (__int128)x * y;
    }
    const long long got = dot_shift<S, n>(a, b);
    const __int128 diff = ((__int128)got * ((__int128)1 << (S - 1))) * 2 - exact;
    worst = std::fmax(worst, std::fabs((double)diff) * std::ldexp(1.0, -S));
  }
  std::printf("dot %d %d %.6f\n", S, n, worst);
}

int main() {
  std::mt19937_64 rng(5);
  dots<64, 1>(rng);
  dots<64, 2>(rng);
  dots<64, 4>(rng);
  dots<63, 1>(rng);
  dots<63, 3>(rng);
  dots<62, 3>(rng);
  std::printf("split %lld %lld\n", bad_split, n_split);
  bool ok[4];
  for (int m = 1; m <= 4; ++m) {
    Rates r;
    const double s9 = m == 4 ? 2.0 : 1.0 / (3 * 0.0036 + 0.5);
    r.s9 = r.s13 = s9;
    r.omegepsl = m == 1 ? 0.0 : 3.0;
    r.omegepslj = m == 1 ? -475.0 / 63.0 : -5.5;
    r.omegxx = m == 1 ? 0.0 : -0.5;
    if (m == 1) { r.s1 = 1.19; r.s2 = 1.4; r.s4 = 1.2; r.s10 = 1.4; r.s16 = 1.98; }
    else if (m == 3) { r.s1 = r.s2 = r.s10 = r.s16 = 1.8; r.s4 = s9; }
    else r.s1 = r.s2 = r.s4 = r.s10 = r.s16 = s9;
    ok[m - 1] = rates_t<double>(r).int_ok;
  }
  std::printf("rates %d %d %d %d\n", ok[0], ok[1], ok[2], ok[3]);
  return 0;
}
