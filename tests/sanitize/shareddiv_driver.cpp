// Host check of the FP64 build's division by a shared reciprocal
// (exo::SharedDiv in exocubed_b200/csrc/exo_internal.h, the same host/device
// code the kernels run): SharedDiv(b)(a) is the IEEE quotient a / b bit for
// bit, for random significands over its range of exponents, denominators of
// all ones and powers of two, quotients placed next to representable numbers
// and next to midpoints, and zeros (in value).  Exit status 0 when all hold.
#include <cmath>
#include <cstdint>
#include <cstdio>
#include <cstring>
#include <random>

#include "../../exocubed_b200/csrc/exo_internal.h"

static double from_bits(uint64_t u) {
  double x;
  std::memcpy(&x, &u, sizeof(x));
  return x;
}
static uint64_t bits(double x) {
  uint64_t u;
  std::memcpy(&u, &x, sizeof(u));
  return u;
}

static long bad = 0, count = 0;
static void check(const exo::SharedDiv& d, double a) {
  const double got = d(a), want = a / d.b;
  ++count;
  if (bits(got) != bits(want) && !(std::isnan(got) && std::isnan(want))) {
    if (bad++ < 10) std::printf("%a / %a = %a, want %a\n", a, d.b, got, want);
  }
}

int main() {
  std::mt19937_64 rng(7);
  auto value = [&](int lo, int hi) {  // random significand, exponent in [lo, hi]
    const uint64_t e = 1023 + lo + (int64_t)(rng() % (uint64_t)(hi - lo + 1));
    return from_bits((rng() & 0x800fffffffffffffull) | (e << 52));
  };
  for (int k = 0; k < 40000; ++k) {
    double b = value(-60, 60);
    if (k % 8 == 1) b = from_bits(bits(b) | 0x000fffffffffffffull);  // all ones
    if (k % 8 == 2) b = from_bits(bits(b) & 0xfff0000000000000ull);  // power of two
    if (k % 8 == 3) b = value(-400, 400);
    if (k % 8 == 4) b = from_bits((bits(b) & 0xfff0000000000000ull) | (rng() % 64));
    const exo::SharedDiv d(b);
    for (int m = 0; m < 80; ++m) check(d, value(-60, 60));
    for (int m = 0; m < 20; ++m) check(d, value(-500, 500));
    if (d(0.) != 0. || d(-0.) != 0.) ++bad;
    // numerators next to q b and to the midpoints (q + ulp/2) b
    for (int m = 0; m < 40; ++m) {
      const double q = value(-60, 60);
      const double a = q * b;
      check(d, a);
      check(d, std::nextafter(a, 1e300));
      check(d, std::nextafter(a, -1e300));
      const double h = (q + 0.5 * (std::nextafter(q, 1e300) - q)) * b;
      check(d, h);
      check(d, (double)((long double)q * b + 0.5L * ((long double)std::nextafter(q, 1e300) - q) * b));
    }
  }
  if (bad) {
    std::printf("shareddiv: %ld of %ld differ\n", bad, count);
    return 1;
  }
  std::printf("shareddiv: ok (%ld)\n", count);
  return 0;
}
