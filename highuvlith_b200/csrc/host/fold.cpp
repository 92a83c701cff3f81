// Kernel sets of real masks (host, FP64).
//
// A real mask has M(-f) = conj M(f).  Where the transmission
// cross-coefficients are real and even under point inversion (a source
// symmetric under inversion, a pupil without phase: every in-focus scalar
// pupil), each eigenspace has a basis of functions w with w(-f) = conj w(f),
// whose fields on a real mask are real.  Two such kernels are then one complex
// transform: with p = w_a + i w_b, |IFFT(p M)|^2 = E_a^2 + E_b^2, so K
// kernels become ceil(K / 2) and the field pass halves.
//
// The eigenvectors come with arbitrary phases and, within an eigenvalue
// cluster, arbitrarily mixed, so the basis is recovered cluster by cluster:
// kernel kappa splits into kappa = a + i b with a(-f) = conj a(f), likewise b;
// the 2 d functions of a cluster of d kernels span d dimensions over the
// reals, and the leading eigenvectors of their Gram matrix give d functions w
// with sum w^2 = sum (a^2 + b^2) for every real mask.  A set whose clusters do
// not have that rank (defocus, an asymmetric source) is left as it is.
//
// Whole calls before and after: 256 clips of 1024^2 (31 kernels as 16) 1.010 ->
// 0.768 ms, 27 of 512^2 (48 kernels) 0.172 -> 0.127 ms, 6 of 2048^2 (64)
// 0.434 -> 0.319 ms.  A new engine folds in its first call on real masks: 0.5 ms
// for 31 kernels of h = 37, 5 ms for 64 of h = 94.
#include <algorithm>
#include <atomic>
#include <cmath>
#include <exception>
#include <mutex>

#include "host.hpp"

namespace huv {

namespace {

// Eigen-decomposition of a small symmetric matrix (row-major n x n) by cyclic
// Jacobi rotations: eigenvalues in d, eigenvectors in the columns of u.
void jacobi(int n, std::vector<double>& a, std::vector<double>& d, std::vector<double>& u) {
  u.assign(static_cast<size_t>(n) * n, 0.0);
  for (int i = 0; i < n; ++i) u[i * n + i] = 1.0;
  for (int sweep = 0; sweep < 60; ++sweep) {
    double off = 0.0, diag = 0.0;
    for (int i = 0; i < n; ++i) {
      diag += a[i * n + i] * a[i * n + i];
      for (int j = i + 1; j < n; ++j) off += a[i * n + j] * a[i * n + j];
    }
    if (off <= 1e-34 * diag) break;
    for (int p = 0; p < n; ++p)
      for (int q = p + 1; q < n; ++q) {
        const double apq = a[p * n + q];
        if (apq == 0.0) continue;
        const double th = (a[q * n + q] - a[p * n + p]) / (2.0 * apq);
        const double t = (th >= 0 ? 1.0 : -1.0) / (std::fabs(th) + std::sqrt(th * th + 1.0));
        const double c = 1.0 / std::sqrt(t * t + 1.0), s = t * c;
        for (int k = 0; k < n; ++k) {
          const double x = a[k * n + p], y = a[k * n + q];
          a[k * n + p] = c * x - s * y;
          a[k * n + q] = s * x + c * y;
        }
        for (int k = 0; k < n; ++k) {
          const double x = a[p * n + k], y = a[q * n + k];
          a[p * n + k] = c * x - s * y;
          a[q * n + k] = s * x + c * y;
        }
        for (int k = 0; k < n; ++k) {
          const double x = u[k * n + p], y = u[k * n + q];
          u[k * n + p] = c * x - s * y;
          u[k * n + q] = s * x + c * y;
        }
      }
  }
  d.resize(n);
  for (int i = 0; i < n; ++i) d[i] = a[i * n + i];
}

// Clusters join eigenvalues this close (relative): the eigenvectors of wider
// gaps are separate to 1e-16 / gap, far below kEnergy.
constexpr double kCluster = 1e-5;
// Energy, of the set's, that the dropped half of a cluster's functions may hold.
constexpr double kEnergy = 1e-13;
constexpr int kMaxCluster = 32;

// Inner product over the whole band of two functions held on half the orders.
double dot(const cd* x, const cd* y, size_t H) {
  double s = 0.0;
  for (size_t o = 0; o < H; ++o)
    s += (o + 1 == H ? 1.0 : 2.0) * (x[o].real() * y[o].real() + x[o].imag() * y[o].imag());
  return s;
}

// dot() of every pair of m functions, side by side: a sum is a chain of
// dependent additions, and clusters of one or two kernels are most of a set.
template <int m>
void gram(const cd* v, size_t H, double* g) {
  double s[m][m] = {};
  for (size_t o = 0; o < H; ++o) {
    const double weight = o + 1 == H ? 1.0 : 2.0;
    for (int p = 0; p < m; ++p)
      for (int q = p; q < m; ++q) {
        const cd x = v[p * H + o], y = v[q * H + o];
        s[p][q] += weight * (x.real() * y.real() + x.imag() * y.imag());
      }
  }
  for (int p = 0; p < m; ++p)
    for (int q = p; q < m; ++q) g[p * m + q] = g[q * m + p] = s[p][q];
}

// body(lo, hi) over [0, n): on the worker threads where the work (doubles
// touched) is worth waking them, about 0.1 ms, else here.
template <typename F>
void each(int64_t n, size_t work, const F& body) {
  if (work < (size_t(1) << 16)) {
    body(0, n);
    return;
  }
  std::exception_ptr failed;  // the workers' first (out of memory)
  std::mutex mu;
  // parallel_for hands out runs of at least 64
  parallel_for(64 * n, [&](int64_t lo, int64_t hi) {
    try {
      body((lo + 63) / 64, (hi + 63) / 64);
    } catch (...) {
      std::lock_guard<std::mutex> lock(mu);
      failed = std::current_exception();
    }
  });
  if (failed) std::rethrow_exception(failed);
}

}  // namespace

namespace {

// The real-field kernels of the first K, on half the orders: w[k][H] (complex
// pairs).  False where the set has no such basis.
bool real_field_kernels(const KernelSet& ks, int K, double div, std::unique_ptr<double[]>& w) {
  const int n = ks.n, h = ks.band_half_width(), B = 2 * h + 1;
  const int S = static_cast<int>(ks.support.size());
  if (K < 2 || 2 * h >= n) return false;  // an order and its inverse must be different bins
  const size_t BB = static_cast<size_t>(B) * B, H = (BB + 1) / 2;  // o and BB - 1 - o are inverse orders
  const std::vector<uint32_t> pos = ks.band_positions();
  double total = 0.0;
  for (int k = 0; k < K; ++k) total += ks.eigenvalues[k] / div;
  const double n2 = static_cast<double>(n) * n;
  w.reset(new double[2 * static_cast<size_t>(K) * H]);
  std::vector<int> first;                          // of every cluster, then K
  for (int k = 0; k < K; ++k)
    if (k == 0 || ks.eigenvalues[k - 1] - ks.eigenvalues[k] > kCluster * ks.eigenvalues[k - 1]) first.push_back(k);
  const int clusters = static_cast<int>(first.size());
  first.push_back(K);
  // (dense and v: the caller's scratch, kept from cluster to cluster)
  auto fold_cluster = [&](int k0, int k1, std::vector<cd>& dense, std::vector<cd>& v) {
    const int d = k1 - k0, m = 2 * d;
    if (d > kMaxCluster) return false;
    dense.assign(BB, cd(0.0, 0.0));
    if (v.size() < m * H) v.resize(m * H);
    for (int k = k0; k < k1; ++k) {
      // every kernel has the set's support, so the next one overwrites it
      const double sc = std::sqrt(ks.eigenvalues[k] / div);
      for (int t = 0; t < S; ++t) dense[pos[t]] = sc * ks.values[static_cast<size_t>(k) * S + t];
      cd* a = &v[static_cast<size_t>(2 * (k - k0)) * H];
      cd* b = a + H;
      for (size_t o = 0; o < H; ++o) {
        const cd x = dense[o], y = dense[BB - 1 - o];  // kappa(f), kappa(-f)
        a[o] = cd(0.5 * (x.real() + y.real()), 0.5 * (x.imag() - y.imag()));
        b[o] = cd(0.5 * (x.imag() + y.imag()), -0.5 * (x.real() - y.real()));
      }
    }
    std::vector<double> g(static_cast<size_t>(m) * m), ev, u;
    if (m == 2)
      gram<2>(v.data(), H, g.data());
    else if (m == 4)
      gram<4>(v.data(), H, g.data());
    else
      for (int p = 0; p < m; ++p)
        for (int q = p; q < m; ++q) g[p * m + q] = g[q * m + p] = dot(&v[p * H], &v[q * H], H);
    jacobi(m, g, ev, u);
    std::vector<int> order(m);
    for (int i = 0; i < m; ++i) order[i] = i;
    std::sort(order.begin(), order.end(), [&](int x, int y) { return ev[x] > ev[y]; });
    double dropped = 0.0;
    for (int i = d; i < m; ++i) dropped += std::fabs(ev[order[i]]);
    if (!(dropped <= kEnergy * total / K * d)) return false;
    for (int j = 0; j < d; ++j) {
      double* out = &w[2 * static_cast<size_t>(k0 + j) * H];
      for (int i = 0; i < m; ++i) {
        const double c = u[i * m + order[j]] / n2;
        const double* x = reinterpret_cast<const double*>(&v[i * H]);
        if (i == 0)
          for (size_t o = 0; o < 2 * H; ++o) out[o] = c * x[o];
        else
          for (size_t o = 0; o < 2 * H; ++o) out[o] += c * x[o];
      }
    }
    return true;
  };
  // the first cluster alone: it already tells an unsuitable set (defocus)
  {
    std::vector<cd> dense, v;
    if (!fold_cluster(first[0], first[1], dense, v)) return false;
  }
  std::atomic<bool> ok{true};
  each(clusters - 1, static_cast<size_t>(K) * BB, [&](int64_t lo, int64_t hi) {
    std::vector<cd> dense, v;
    for (int64_t c = lo; c < hi && ok; ++c)
      if (!fold_cluster(first[c + 1], first[c + 2], dense, v)) ok = false;
  });
  return ok;
}

// Kernels 2 f and 2 f + 1 as one: x + i y, in whole bands.
template <typename T>
void pair_kernels(const double* w, int K, size_t BB, T* out) {
  const size_t H = (BB + 1) / 2;
  const int F = (K + 1) / 2;
  each(F, static_cast<size_t>(K) * BB, [&](int64_t lo, int64_t hi) {
    for (int64_t f = lo; f < hi; ++f) {
      const double* x = &w[4 * static_cast<size_t>(f) * H];
      const double* y = 2 * f + 1 < K ? x + 2 * H : nullptr;
      T* p = &out[2 * f * BB];
      for (size_t o = 0; o < H; ++o) {
        const double xr = x[2 * o], xi = x[2 * o + 1], yr = y ? y[2 * o] : 0.0, yi = y ? y[2 * o + 1] : 0.0;
        p[2 * o] = static_cast<T>(xr - yi);  // x + i y
        p[2 * o + 1] = static_cast<T>(xi + yr);
        p[2 * (BB - 1 - o)] = static_cast<T>(xr + yi);  // conj x + i conj y
        p[2 * (BB - 1 - o) + 1] = static_cast<T>(yr - xi);
      }
    }
  });
}

template <typename T>
bool fold(const KernelSet& ks, int K, double div, std::unique_ptr<T[]>& v, size_t& size) {
  std::unique_ptr<double[]> w;
  if (!real_field_kernels(ks, K, div, w)) return false;
  const size_t B = 2 * static_cast<size_t>(ks.band_half_width()) + 1;
  size = static_cast<size_t>((K + 1) / 2) * B * B;
  v.reset(new T[2 * size]);
  pair_kernels(w.get(), K, B * B, v.get());
  return true;
}

}  // namespace

bool fold_real_kernels(const KernelSet& ks, int K, double div, FoldedKernels& folded) {
  return fold(ks, K, div, folded.v, folded.size);
}

bool fold_real_kernels(const KernelSet& ks, int K, double div, std::unique_ptr<float[]>& v, size_t& size) {
  return fold(ks, K, div, v, size);
}

}  // namespace huv
