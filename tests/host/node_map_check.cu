// div_by against / and %, over divisors and dividends below 2^31 (run on the
// host): multiples of the divisor and their neighbours, the range's ends and
// a stride through it.  Prints the divisors tried and the wrong results.
#include <cstdint>
#include <cstdio>

#include "lbm_internal.cuh"

int main() {
  long long bad = 0, divisors = 0;
  auto one = [&](uint32_t n, int d, unsigned inv) {
    int rem;
    const int q = lbm::div_by(n, d, inv, rem);
    bad += q != (int)(n / (uint32_t)d) || rem != (int)(n % (uint32_t)d);
  };
  for (long long d = 1; d < (1LL << 31); d += d < 2100 ? 1 : d / 3) {
    const unsigned inv = lbm::div_inv((int)d);
    ++divisors;
    for (long long k = 0; k <= 400; ++k) {
      const long long top = 0x7fffffffLL / d;
      for (long long m : {k, top - k})
        for (long long e = -1; e <= 1; ++e) {
          const long long n = m * d + e;
          if (n >= 0 && n <= 0x7fffffffLL) one((uint32_t)n, (int)d, inv);
        }
      one((uint32_t)(k * 5368709LL), (int)d, inv);
    }
  }
  std::printf("%lld %lld\n", divisors, bad);
  return 0;
}
