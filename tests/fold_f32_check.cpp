// Host check of the FP32 folded kernels (csrc/host/fold.cpp): the FP64 ones
// rounded, bit for bit, and band_positions() against the orders themselves,
// with the worker threads and without.  Prints: K folded differing misplaced.
#include <cstdio>

#include "../highuvlith_b200/csrc/host/host.hpp"
using namespace huv;

int main() {
  for (int n : {64, 256}) {
    Fill f;
    f.kind = HUV_FILL_ANNULAR;
    f.p[0] = 0.4;
    f.p[1] = 0.8;
    f.prepare();
    Optics o;
    o.kind = HUV_OPTICS_EUV;
    o.na = 0.33;
    o.medium = 1.0;
    const auto pts = sample_source(f, 9, 1.0 / (n * 4.0) / o.cutoff(13.5));
    const KernelSet ks = build_kernels(pts, o, n, 4.0, 13.5, 40, 1.0, 0.0);
    const int h = ks.band_half_width(), B = 2 * h + 1;
    int misplaced = 0;
    const auto pos = ks.band_positions();
    for (size_t t = 0; t < pos.size(); ++t) {
      const int my = static_cast<int>(pos[t]) / B - h, mx = static_cast<int>(pos[t]) % B - h;
      misplaced += ks.support[t] != static_cast<int64_t>((my + n) % n) * n + (mx + n) % n;
    }
    for (int K : {2, 3, ks.num_kernels()}) {
      FoldedKernels d;
      std::unique_ptr<float[]> v;
      size_t size = 0;
      const bool a = fold_real_kernels(ks, K, 1.3, d), b = fold_real_kernels(ks, K, 1.3, v, size);
      int differing = a != b || (a && size != d.size);
      for (size_t i = 0; a && b && i < 2 * size; ++i) differing += v[i] != static_cast<float>(d.v[i]);
      printf("%d %d %d %d\n", K, a ? 1 : 0, differing, misplaced);
    }
  }
  return 0;
}
