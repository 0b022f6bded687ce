// quotient() (sih26_b200/csrc/quotient.cuh) against the host's IEEE division, bit for bit: divisors of every
// binary exponent with random, empty and full mantissas, dividends over the whole range, its ends, zeros,
// infinities and NaN. Prints ok, or the first pair that differs. Run by tests/test_quotient_cpu.py.
#include <cfloat>
#include <cmath>
#include <cstdint>
#include <cstdio>
#include <cstring>
#include <initializer_list>
#include <random>

#include "quotient.cuh"

static uint64_t bits(double v) {
  uint64_t u;
  std::memcpy(&u, &v, 8);
  return u;
}
static double make(uint64_t sign, uint64_t exponent, uint64_t mantissa) {
  const uint64_t u = sign << 63 | exponent << 52 | (mantissa & ((1ull << 52) - 1));
  double v;
  std::memcpy(&v, &u, 8);
  return v;
}
static bool same(double a, double b) {
  const double got = sih26::quotient(a, b, sih26::quotient_reciprocal(b)), want = a / b;
  if (bits(got) == bits(want) || (got != got && want != want)) return true;
  std::printf("%a / %a: %a, not %a\n", a, b, got, want);
  return false;
}

int main() {
  std::mt19937_64 rng(20260826);
  const uint64_t full = ~0ull;
  for (uint64_t eb = 0; eb < 2047; ++eb)
    for (int k = 0; k < 600; ++k) {
      const uint64_t mb = k % 3 == 0 ? rng() : k % 3 == 1 ? full - rng() % 3 : rng() % 3;
      const double b = make(0, eb, mb);
      if (b == 0.0) continue;
      const uint64_t ea = rng() % 2047;
      const uint64_t ma = k % 2 == 0 ? rng() : k % 4 == 1 ? full - rng() % 3 : rng() % 3;
      if (!same(make(k & 1, ea, ma), b)) return 1;
      // quotients near 1, and next to a product
      if (!same(make(0, eb, ma), b) || !same(b * make(0, 1023, ma), b)) return 1;
    }
  for (double b : {DBL_MIN, 4.9e-324, 1e-60, 1e-41, 1e-40, 1.0, 3.0, 1e40, 1e41, 1e200, DBL_MAX})
    for (double a : {0.0, -0.0, 4.9e-324, DBL_MIN, 1e-310, 1e-295, 1e-290, 1e-250, 1.0, 1e250, 1e300, DBL_MAX,
                     (double)INFINITY, -(double)INFINITY, (double)NAN})
      if (!same(a, b)) return 1;
  std::puts("ok");
  return 0;
}
