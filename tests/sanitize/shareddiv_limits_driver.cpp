// Host check of exo::SharedDiv (exocubed_b200/csrc/exo_internal.h) where its
// correction steps do not apply: zeros of either sign, infinities and NaN as
// numerators and denominators, and quotients past the largest double.  Every
// result is the division's bit for bit (NaN for NaN).  Exit status 0 when all
// hold.
#include <cmath>
#include <cstdint>
#include <cstdio>
#include <cstring>
#include <limits>

#include "../../exocubed_b200/csrc/exo_internal.h"

int main() {
  const double inf = std::numeric_limits<double>::infinity(), nan = std::nan("");
  const double a[] = {0., -0., inf, -inf, nan, 1., -1., 3e100, -7e-100, 0x1p500, -0x1p-500};
  const double b[] = {inf, -inf, 0., -0., nan, 1., -3., 0x1.8p400, -0x1.8p-400, 600., 0.1};
  volatile double top = 0x1p1000, small = 0x1p-400;  // a quotient past the largest double
  long bad = 0, count = 0;
  auto check = [&](double x, double y) {
    const double got = exo::SharedDiv(y)(x), want = x / y;
    uint64_t g, w;
    std::memcpy(&g, &got, 8);
    std::memcpy(&w, &want, 8);
    ++count;
    if (g != w && !(std::isnan(got) && std::isnan(want))) {
      ++bad;
      std::printf("%a / %a = %a, want %a\n", x, y, got, want);
    }
  };
  for (double x : a)
    for (double y : b) check(x, y);
  check(top, small);
  check(-top, small);
  if (bad) {
    std::printf("shareddiv limits: %ld of %ld differ\n", bad, count);
    return 1;
  }
  std::printf("shareddiv limits: ok (%ld)\n", count);
  return 0;
}
