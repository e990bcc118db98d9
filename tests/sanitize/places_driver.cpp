// Host check of the kernels' 32-bit places (exo::geo_place, exo::row_place):
// the same as in 64 bits at the corners of the metric and of the states up to
// the largest grid that view_allocate takes, without signed overflow (run
// under UndefinedBehaviorSanitizer).  Exit status 0 when all hold.
#include <cstdio>
#include <initializer_list>

#include "../../exocubed_b200/csrc/exo_internal.h"

int main() {
  long bad = 0, count = 0;
  for (int nc : {12, 102, 3454, 3456, 3606, 4806, 4884}) {
    if (!exo::places_fit(nc, nc)) ++bad;
    for (int p = 0; p < 6; ++p)
      for (int k : {0, nc / 2, nc - 1})
        for (int j : {0, nc / 2, nc - 1}) {
          for (int f = 0; f < exo::NGEO2D; ++f, ++count)
            if (exo::geo_place(nc, nc, f, p, k, j) != (((size_t)f * 6 + p) * nc + k) * nc + j) ++bad;
          for (int nv : {4, 5})
            for (int n = 0; n < nv; ++n, ++count)
              if (exo::row_place(nv, nc, nc, p, n, k, j) != (((size_t)p * nv + n) * nc + k) * nc + j)
                ++bad;
        }
  }
  if (exo::places_fit(4886, 4886)) ++bad;
  if (bad) {
    std::printf("places: %ld of %ld differ\n", bad, count);
    return 1;
  }
  std::printf("places: ok (%ld)\n", count);
  return 0;
}
