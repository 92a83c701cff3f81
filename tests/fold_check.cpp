// Host check of the kernel sets of real masks (csrc/host/fold.cpp): for each
// source, pupil and kernel count, sum |p M|^2 of the folded kernels against
// sum |kappa M|^2 of the set itself, in FP64, for a random real mask's band at
// random points.  Prints: name K folded max_rel_err.
#include <cmath>
#include <cstdio>
#include <random>

#include "../highuvlith_b200/csrc/host/host.hpp"
using namespace huv;

namespace {

double max_err(const KernelSet& ks, int K, double div, const FoldedKernels& p) {
  const int n = ks.n, h = ks.band_half_width(), B = 2 * h + 1, F = (K + 1) / 2;
  const size_t BB = static_cast<size_t>(B) * B;
  std::mt19937 rng(K + B);
  std::normal_distribution<double> g;
  std::vector<cd> M(BB);
  for (size_t o = 0; o < BB; ++o) M[o] = cd(g(rng), g(rng));
  for (size_t o = 0; o < BB / 2; ++o) M[BB - 1 - o] = std::conj(M[o]);
  M[BB / 2] = M[BB / 2].real();
  double worst = 0, top = 0;
  for (int s = 0; s < 12; ++s) {
    const double x = std::uniform_real_distribution<double>(0, n)(rng), y = std::uniform_real_distribution<double>(0, n)(rng);
    std::vector<cd> e(BB);
    for (int i = 0; i < B; ++i)
      for (int j = 0; j < B; ++j) e[i * B + j] = M[i * B + j] * std::polar(1.0, 2 * M_PI * ((i - h) * y + (j - h) * x) / n);
    double a = 0, b = 0;
    for (int k = 0; k < K; ++k) {
      cd f = 0;
      for (size_t t = 0; t < ks.support.size(); ++t) {
        const int i = ks.support[t] / n, j = ks.support[t] % n;
        const int my = (i < n / 2 ? i : i - n) + h, mx = (j < n / 2 ? j : j - n) + h;
        f += ks.values[k * ks.support.size() + t] * e[my * B + mx];
      }
      a += ks.eigenvalues[k] / div * std::norm(f) / (double(n) * n * n * n);
    }
    for (int k = 0; k < F; ++k) {
      cd f = 0;
      for (size_t o = 0; o < BB; ++o) f += p[k * BB + o] * e[o];
      b += std::norm(f);
    }
    worst = std::fmax(worst, std::fabs(a - b));
    top = std::fmax(top, a);
  }
  return worst / top;
}

void run(const char* name, int kind, std::vector<double> par, double lambda, double na, double obs, int n, double px,
         int kmax, double z) {
  Fill f;
  f.kind = kind;
  for (size_t i = 0; i < par.size(); ++i) f.p[i] = par[i];
  f.prepare();
  Optics o;
  o.kind = lambda < 20 ? HUV_OPTICS_EUV : HUV_OPTICS_PROJECTION;
  o.na = na;
  o.medium = na > 1 ? 1.437 : 1.0;
  o.obscuration = obs;
  const auto pts = sample_source(f, 0, 1.0 / (n * px) / o.cutoff(lambda));
  const KernelSet ks = build_kernels(pts, o, n, px, lambda, kmax, 1.0, z);
  for (int k : {1, 2, 3, 5, 8, 16, kmax}) {
    const int K = std::min(select_kernel_count(ks.all_values.empty() ? ks.eigenvalues : ks.all_values, ks.trace, k, 1.0),
                           ks.num_kernels());
    FoldedKernels p;
    const bool ok = fold_real_kernels(ks, K, 1.7, p);
    printf("%s %d %d %.3e\n", name, K, ok ? 1 : 0, ok ? max_err(ks, K, 1.7, p) : 0.0);
  }
}

}  // namespace

int main() {
  run("conventional", HUV_FILL_CONVENTIONAL, {0.5}, 13.5, 0.33, 0, 64, 4, 32, 0);
  run("annular", HUV_FILL_ANNULAR, {0.6, 0.85}, 193.368, 1.35, 0, 64, 16, 30, 0);
  run("obscured", HUV_FILL_ANNULAR, {0.3, 0.8}, 13.5, 0.55, 0.2, 64, 3, 31, 0);
  run("dipole", HUV_FILL_DIPOLE, {0.8, 0.1, 0.0}, 193.368, 1.35, 0, 64, 16, 24, 0);
  run("dipole30", HUV_FILL_DIPOLE, {0.7, 0.15, 30.0}, 13.5, 0.33, 0, 64, 4, 24, 0);
  run("quadrupole", HUV_FILL_QUADRUPOLE, {0.7, 0.15, 45.0}, 13.5, 0.33, 0, 64, 4, 24, 0);
  run("quasar", HUV_FILL_QUASAR, {0.7, 0.9, 45.0}, 13.5, 0.33, 0, 64, 4, 40, 0);
  run("gaussian", HUV_FILL_GAUSSIAN, {0.4}, 193.368, 0.93, 0, 64, 16, 24, 0);
  run("defocus", HUV_FILL_CONVENTIONAL, {0.5}, 13.5, 0.33, 0, 64, 4, 32, 50);
  run("nyquist", HUV_FILL_CONVENTIONAL, {0.9}, 13.5, 0.33, 0, 32, 14, 16, 0);
  // an asymmetric set: one kernel pair of random values
  KernelSet ks;
  ks.n = 32;
  std::mt19937 rng(1);
  std::normal_distribution<double> g;
  for (int i : {0, 1, 2, 31})
    for (int j : {0, 1, 31}) ks.support.push_back(i * 32 + j);
  ks.eigenvalues = {2.0, 1.0};
  for (size_t i = 0; i < 2 * ks.support.size(); ++i) ks.values.push_back(cd(g(rng), g(rng)));
  FoldedKernels p;
  printf("asymmetric 2 %d 0\n", fold_real_kernels(ks, 2, 1.0, p) ? 1 : 0);
  return 0;
}
