// Host check of csrc/cuda/band_plan.cuh: the room sized for the partial sums of
// the flare mean against the blocks that the column pass and the rectangle
// spectrum launch, restated here.  Prints: n cases short.
#include <cstdio>

#include "../highuvlith_b200/csrc/cuda/band_plan.cuh"
using namespace huv_dev;

int main() {
  for (int n = 8; n <= 8192; n *= 2) {
    int cases = 0, shortfall = 0;
    for (int hb = 0; 2 * hb < n && hb <= 1024; ++hb) {
      const int B = 2 * hb + 1, S = xt_fits(n, hb) ? xt_S(n) : fit_units(4, 2 * sizeof(float2) * size_t(n));
      for (int cols : {B, hb + 1}) {
        ++cases;
        if ((cols + S - 1) / S > band_mean_parts(n, hb)) ++shortfall;
      }
      if (B <= 255 && (B + 15) / 16 > band_mean_parts(n, hb)) ++shortfall;
    }
    printf("%d %d %d\n", n, cases, shortfall);
  }
  return 0;
}
