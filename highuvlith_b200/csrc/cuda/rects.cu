// Exact band spectrum of rectangle clips (HUV_INPUT_RECTS).
//
// Mask::spectrum's closed form (crates/highuvlith-core/src/mask.rs:616-657,
// 1439-1503): a separable term with intervals [a, b] in x and [c, d] in y has
// the FFT-layout coefficient
//     S(ky, kx) = N^2 phi(ky) phi(kx) (g_ky(d) - g_ky(c)) (g_kx(b) - g_kx(a)),
//     g_m(x) = e^{-2 pi i m x / L} / (-2 pi i m)  (m != 0),  g_0(x) = x / L,
//     phi(m) = e^{-i pi m (N - 1) / N}   (pixel-centre sampling, mask.rs:28-36).
// Overlapping rectangles are resolved as the reference's compress does
// (mask.rs:1365-1437): the clip's distinct y edges cut it into rows; each
// row's covered x cells merge into runs.  The union is then
// sum_rows Y_j(ky) X_j(kx), X_j = sum of the row's run terms -- a complex GEMM
// over rows, done on the GPU in FP64.  Clips of up to kRectSortMax rectangles
// are resolved on the GPU:
//   rect_sort: one block per clip clips its rectangles to the field and sorts
//     them by left edge and their y edges, in shared memory;
//   rect_edges: g_m of every left, right and y edge, for every band order;
//   rect_rows: one warp per row walks the sorted rectangles, merges those that
//     cover the row into runs and adds up X_j from the edges' table.
// (40 clips of 60 rectangles at 512^2: the host's resolution took 2.0 of
// 3.4 ms per call, with two synchronous copies; the three kernels take 0.03.)
// Clips with more are resolved on the host (which also merges rows with equal
// runs), and
//   rect_row_coef: one warp per row: X_j(kx) for every band order kx (each
//     lane walks the orders lane, lane + 32, ... by a phasor recurrence from
//     two sincos per run) and Y_j(ky).
// Then
//   rect_band_gemm: per clip and block of band rows ky, M(ky, kx) =
//     (feature - background) sum_j Y_j(ky) X_j(kx) (+ background N^2 at DC),
//     rows staged through shared memory; the block's share of the flare mean
//     sum W |M|^2 goes to a fixed slot (summed in order by mean_reduce).
#include <cuda_runtime.h>
#include <stdint.h>

#include <algorithm>
#include <cmath>
#include <cstring>
#include <vector>

#include "../engine.hpp"
#include "band_plan.cuh"

namespace huv_dev {

struct RectRowDev {
  double y0, y1;
  int32_t first, count;  // runs[first .. first + count)
};

__device__ __forceinline__ double2 zmul(double2 a, double2 b) {
  return make_double2(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x);
}

// Sum over intervals [a_r, b_r] of (g_m(b) - g_m(a)) for m = m0 + 32 i,
// i < cnt, accumulated into acc[i] (L-normalised).
__device__ void run_terms(const double2* __restrict__ runs, int first, int count, double L, int m0, int cnt,
                          double2* acc) {
  const double two_pi = 6.283185307179586476925;
  for (int r = 0; r < count; ++r) {
    const double2 ab = runs[first + r];
    // e^{-2 pi i m x / L} at m = m0 and the step e^{-2 pi i 32 x / L}, x = a, b
    double sa0, ca0, sb0, cb0, sas, cas, sbs, cbs;
    sincospi(-2.0 * m0 * ab.x / L, &sa0, &ca0);
    sincospi(-2.0 * m0 * ab.y / L, &sb0, &cb0);
    sincospi(-64.0 * ab.x / L, &sas, &cas);
    sincospi(-64.0 * ab.y / L, &sbs, &cbs);
    double2 ea = make_double2(ca0, sa0), eb = make_double2(cb0, sb0);
    const double2 sa = make_double2(cas, sas), sb = make_double2(cbs, sbs);
    for (int i = 0; i < cnt; ++i) {
      const int m = m0 + 32 * i;
      if (m == 0) {
        acc[i].x += (ab.y - ab.x) / L;
      } else {
        // (eb - ea) / (-2 pi i m) = i (eb - ea) / (2 pi m)
        const double f = 1.0 / (two_pi * m);
        acc[i].x += -(eb.y - ea.y) * f;
        acc[i].y += (eb.x - ea.x) * f;
      }
      ea = zmul(ea, sa);
      eb = zmul(eb, sb);
    }
  }
}

// X[j][m + h] and Y[j][m + h] for every row j (one warp per row).
__global__ void rect_row_coef(const RectRowDev* __restrict__ rows, const double2* __restrict__ runs, int n_rows,
                              int h, double L, double2* __restrict__ X, double2* __restrict__ Y) {
  const int warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
  if (warp >= n_rows) return;
  const int B = 2 * h + 1;
  const int m0 = -h + lane;
  const int cnt = m0 <= h ? (h - m0) / 32 + 1 : 0;
  double2 ax[8], ay[8];  // B <= 255 -> at most 8 orders per lane
#pragma unroll
  for (int i = 0; i < 8; ++i) ax[i] = ay[i] = make_double2(0.0, 0.0);
  const RectRowDev rw = rows[warp];
  if (cnt > 0) {
    run_terms(runs, rw.first, rw.count, L, m0, cnt, ax);
    const double2 yr = make_double2(rw.y0, rw.y1);
    run_terms(&yr, 0, 1, L, m0, cnt, ay);
  }
  for (int i = 0; i < cnt; ++i) {
    const int k = m0 + 32 * i + h;
    X[static_cast<size_t>(warp) * B + k] = ax[i];
    Y[static_cast<size_t>(warp) * B + k] = ay[i];
  }
}

// ------------------------------------------------ resolution on the device
constexpr int kRectSortMax = 2048;  // rectangles per clip

// Bitonic sort of n (a power of two) keys in shared memory, with their values.
template <bool VAL>
__device__ void bitonic(double* key, int16_t* val, int n) {
  for (int k = 2; k <= n; k <<= 1)
    for (int j = k >> 1; j > 0; j >>= 1) {
      __syncthreads();
      for (int i = threadIdx.x; i < n / 2; i += blockDim.x) {
        const int a = 2 * j * (i / j) + i % j, b = a + j;
        const bool up = (a & k) == 0;
        const double x = key[a], y = key[b];
        if ((x > y) == up) {
          key[a] = y;
          key[b] = x;
          if (VAL) {
            const int16_t t = val[a];
            val[a] = val[b];
            val[b] = t;
          }
        }
      }
    }
  __syncthreads();
}

// First rectangle of clip c and the clip's count.  Held within the `total`
// rectangles that the tables are sized for: a caller's graph that captured a
// call may be launched after other calls have brought other offsets.
__device__ __forceinline__ int2 rect_span(const int32_t* __restrict__ offs, int c, int total) {
  const int o0 = min(max(offs[c] - offs[0], 0), total);
  return make_int2(o0, min(max(offs[c + 1] - offs[c], 0), total - o0));
}

// One block per clip: its rectangles, clipped to the field and with empty
// ones left out, sorted by left edge into sorted[o0 ..], its distinct y edges
// ascending into ys[2 o0 ..], and the counts (rectangles, edges).  Absent
// entries sort as +infinity.  Shared memory: keys [2 cap], values [cap], cap =
// the power of two that holds the largest clip.
__global__ void __launch_bounds__(256) rect_sort(const double* __restrict__ rects, const int32_t* __restrict__ offs,
                                                  int total, double half, int cap, double4* __restrict__ sorted,
                                                  double* __restrict__ ys, int2* __restrict__ counts) {
  extern __shared__ double rsm[];
  double* key = rsm;                                          // [2 cap]
  int16_t* val = reinterpret_cast<int16_t*>(key + 2 * cap);  // [cap]
  __shared__ int s_n;
  const double inf = __longlong_as_double(0x7ff0000000000000ll);
  const int c = blockIdx.x;
  const int2 span = rect_span(offs, c, total);
  const int o0 = span.x, n = min(span.y, cap);
  const double* q = rects + 4 * static_cast<size_t>(o0);
  auto rect = [&](int i) {
    return make_double4(fmax(q[4 * i] - q[4 * i + 2] / 2.0, -half), fmin(q[4 * i] + q[4 * i + 2] / 2.0, half),
                        fmax(q[4 * i + 1] - q[4 * i + 3] / 2.0, -half), fmin(q[4 * i + 1] + q[4 * i + 3] / 2.0, half));
  };
  int p2 = 1;
  while (p2 < n) p2 <<= 1;
  if (threadIdx.x == 0) s_n = 0;
  __syncthreads();
  for (int i = threadIdx.x; i < p2; i += blockDim.x) {
    double k = inf;
    if (i < n) {
      const double4 r = rect(i);
      if (r.y > r.x && r.w > r.z) {
        k = r.x;
        atomicAdd(&s_n, 1);
      }
    }
    key[i] = k;
    val[i] = static_cast<int16_t>(i);
  }
  bitonic<true>(key, val, p2);
  const int live = s_n;
  for (int i = threadIdx.x; i < live; i += blockDim.x) sorted[o0 + i] = rect(val[i]);
  __syncthreads();
  for (int i = threadIdx.x; i < 2 * p2; i += blockDim.x) {
    double k = inf;
    if (i / 2 < n) {
      const double4 r = rect(i / 2);
      if (r.y > r.x && r.w > r.z) k = (i & 1) ? r.w : r.z;
    }
    key[i] = k;
  }
  bitonic<false>(key, nullptr, 2 * p2);
  // distinct edges, in order (one warp)
  if (threadIdx.x < 32) {
    int m = 0;
    for (int b = 0; b < 2 * live; b += 32) {
      const int i = b + threadIdx.x;
      const bool keep = i < 2 * live && (i == 0 || key[i] != key[i - 1]);
      const unsigned mask = __ballot_sync(0xffffffffu, keep);
      if (keep) ys[2 * static_cast<size_t>(o0) + m + __popc(mask & ((1u << threadIdx.x) - 1))] = key[i];
      m += __popc(mask);
    }
    if (threadIdx.x == 0) counts[c] = make_int2(live, m);
  }
}

// g_m(x) = e^{-2 pi i m x / L} / (-2 pi i m), g_0 = x / L, for every order of
// the band: EX[rect][left, right][B], EY[y edge][B].  One thread per value.
__global__ void __launch_bounds__(256) rect_edges(const int32_t* __restrict__ offs, int rects, const int2* __restrict__ counts,
                                                   const double4* __restrict__ sorted, const double* __restrict__ ys,
                                                   int h, double L, double2* __restrict__ EX,
                                                   double2* __restrict__ EY) {
  const int c = blockIdx.y, o0 = rect_span(offs, c, rects).x, B = 2 * h + 1;
  const int2 n = counts[c];
  const int nx = 2 * n.x, total = (nx + n.y) * B;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < total; i += gridDim.x * blockDim.x) {
    const int e = i / B, k = i - e * B, m = k - h;
    const double4 r = e < nx ? sorted[o0 + e / 2] : make_double4(0, 0, 0, 0);
    const double x = e < nx ? ((e & 1) ? r.y : r.x) : ys[2 * static_cast<size_t>(o0) + e - nx];
    double2 g = make_double2(x / L, 0.0);
    if (m != 0) {
      double s, co;
      sincospi(-2.0 * m * x / L, &s, &co);
      const double f = 1.0 / (6.283185307179586476925 * m);  // 1 / (-2 pi i m) = i / (2 pi m)
      g = make_double2(-s * f, co * f);
    }
    (e < nx ? EX + (static_cast<size_t>(2 * o0) + e) * B : EY + (static_cast<size_t>(2 * o0) + e - nx) * B)[k] = g;
  }
}

// One warp per row j of a clip (between its y edges j and j + 1): X[j][m] =
// sum over the row's runs of g(right) - g(left), Y[j][m] = g(y_j+1) - g(y_j).
// A run grows while the next covering rectangle starts at or before its end.
__global__ void __launch_bounds__(256) rect_rows(const int32_t* __restrict__ offs, int rects, const int2* __restrict__ counts,
                                                  const double4* __restrict__ sorted, const double* __restrict__ ys,
                                                  const double2* __restrict__ EX, const double2* __restrict__ EY, int h,
                                                  double2* __restrict__ X, double2* __restrict__ Y) {
  const int c = blockIdx.y, o0 = rect_span(offs, c, rects).x, B = 2 * h + 1, lane = threadIdx.x & 31;
  const int2 n = counts[c];
  const size_t e0 = 2 * static_cast<size_t>(o0);
  for (int j = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; j + 1 < n.y; j += (gridDim.x * blockDim.x) >> 5) {
    const double ya = ys[e0 + j], yb = ys[e0 + j + 1];
    double2 acc[8];  // B <= 255: orders lane, lane + 32, ...
#pragma unroll
    for (int i = 0; i < 8; ++i) acc[i] = make_double2(0.0, 0.0);
    auto add = [&](int a, int b) {  // the run from rectangle a's left to b's right edge
      const double2 *ga = EX + (e0 + 2 * a) * B, *gb = EX + (e0 + 2 * b + 1) * B;
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        const int k = lane + 32 * i;
        if (k < B) {
          acc[i].x += gb[k].x - ga[k].x;
          acc[i].y += gb[k].y - ga[k].y;
        }
      }
    };
    int first = -1, last = -1;  // rectangles of the run's left edge and furthest right edge
    double end = 0.0;
    for (int b = 0; b < n.x; b += 32) {
      const int r = b + lane;
      const double4 q = r < n.x ? sorted[o0 + r] : make_double4(0.0, 0.0, 1.0, 0.0);
      unsigned mask = __ballot_sync(0xffffffffu, r < n.x && q.z <= ya && q.w >= yb);
      while (mask) {
        const int s = __ffs(mask) - 1;
        mask &= mask - 1;
        const double x0 = __shfl_sync(0xffffffffu, q.x, s), x1 = __shfl_sync(0xffffffffu, q.y, s);
        if (first >= 0 && x0 > end) {
          add(first, last);
          first = -1;
        }
        if (first < 0) {
          first = last = b + s;
          end = x1;
        } else if (x1 > end) {
          last = b + s;
          end = x1;
        }
      }
    }
    if (first >= 0) add(first, last);
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const int k = lane + 32 * i;
      if (k < B) {
        X[(e0 + j) * B + k] = acc[i];
        const double2 g0 = EY[(e0 + j) * B + k], g1 = EY[(e0 + j + 1) * B + k];
        Y[(e0 + j) * B + k] = make_double2(g1.x - g0.x, g1.y - g0.y);
      }
    }
  }
}

// M(ky, kx) for clip c0 + blockIdx.y, band rows ky in [blockIdx.x * TY, +TY).
// Thread t owns (ky, kx) pairs t, t + 256, ... of the tile; rows staged 16 at
// a time.  Dynamic shared memory: 16 * (TY + B) double2.
// The rows of clip c are clip_rows[c] .. clip_rows[c + 1] (resolved on the
// host), or, with `counts`, the counts[c].y - 1 rows from twice the clip's first
// rectangle on (clip_rows = the offsets of the clips among `rects` rectangles).
__global__ void __launch_bounds__(256) rect_band_gemm(const int32_t* __restrict__ clip_rows, int rects,
                                                       const int2* __restrict__ counts, const double2* __restrict__ X, const double2* __restrict__ Y,
                                                       int c0, int h, int n, double2 dv, double2 bgn2,
                                                       const float* __restrict__ W, float2* __restrict__ Mband,
                                                       float* __restrict__ parts) {
  extern __shared__ double2 rs[];
  constexpr int TY = kRectTY, MAXE = (TY * 255 + 255) / 256;
  const int B = 2 * h + 1;
  const int clip = blockIdx.y, cg = c0 + clip;
  const int ky0 = blockIdx.x * TY;
  const int ty = min(TY, B - ky0);
  double2* sy = rs;               // [16][TY]
  double2* sx = rs + 16 * TY;     // [16][B]
  const int j0 = counts ? 2 * rect_span(clip_rows, cg, rects).x : clip_rows[cg];
  const int j1 = counts ? j0 + max(counts[cg].y - 1, 0) : clip_rows[cg + 1];
  const int nout = ty * B;
  double2 acc[MAXE];
#pragma unroll
  for (int e = 0; e < MAXE; ++e) acc[e] = make_double2(0.0, 0.0);
  for (int jb = j0; jb < j1; jb += 16) {
    const int nj = min(16, j1 - jb);
    __syncthreads();
    for (int t = threadIdx.x; t < nj * B; t += blockDim.x) {
      const int jj = t / B, k = t - jj * B;
      sx[jj * B + k] = X[static_cast<size_t>(jb + jj) * B + k];
    }
    for (int t = threadIdx.x; t < nj * ty; t += blockDim.x) {
      const int jj = t / ty, k = t - jj * ty;
      sy[jj * TY + k] = Y[static_cast<size_t>(jb + jj) * B + ky0 + k];
    }
    __syncthreads();
#pragma unroll
    for (int e = 0; e < MAXE; ++e) {
      const int o = threadIdx.x + 256 * e;
      if (o < nout) {
        const int r = o / B, kx = o - r * B;
        double2 a = acc[e];
        for (int jj = 0; jj < nj; ++jj) {
          const double2 yv = sy[jj * TY + r], xv = sx[jj * B + kx];
          a.x = fma(yv.x, xv.x, fma(-yv.y, xv.y, a.x));
          a.y = fma(yv.x, xv.y, fma(yv.y, xv.x, a.y));
        }
        acc[e] = a;
      }
    }
  }
  // scale, DC, store, flare-mean partial
  __shared__ float red[8];
  float wsum = 0.f;
  const double n2 = static_cast<double>(n) * n;
#pragma unroll
  for (int e = 0; e < MAXE; ++e) {
    const int o = threadIdx.x + 256 * e;
    if (o < nout) {
      const int r = o / B, kx = o - r * B;
      const int my = ky0 + r;
      const int qy = my - h, qx = kx - h;
      // N^2 phi(qy) phi(qx), phi(m) = e^{-i pi m (N - 1) / N}
      double s, c;
      sincospi(-static_cast<double>(qy + qx) * (n - 1) / n, &s, &c);
      const double2 ph = make_double2(c * n2, s * n2);
      double2 v = zmul(zmul(acc[e], ph), dv);
      if (qy == 0 && qx == 0) {
        v.x += bgn2.x;
        v.y += bgn2.y;
      }
      const float2 f = make_float2(static_cast<float>(v.x), static_cast<float>(v.y));
      Mband[(static_cast<size_t>(clip) * B + my) * B + kx] = f;
      if (W) wsum += W[my * B + kx] * (f.x * f.x + f.y * f.y);
    }
  }
  if (parts) {
    for (int o = 16; o > 0; o >>= 1) wsum += __shfl_xor_sync(0xffffffffu, wsum, o);
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = wsum;
    __syncthreads();
    if (threadIdx.x == 0) {
      float t = 0.f;
      for (int w = 0; w < 8; ++w) t += red[w];
      parts[static_cast<size_t>(clip) * gridDim.x + blockIdx.x] = t;
    }
  }
}

// mean[c] = sum_i parts[c][i] in order (deterministic).
__global__ void rect_mean_reduce(const float* __restrict__ parts, int nparts, int clips, float* __restrict__ mean) {
  const int c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= clips) return;
  float s = 0.f;
  for (int i = 0; i < nparts; ++i) s += parts[static_cast<size_t>(c) * nparts + i];
  mean[c] = s;
}

}  // namespace huv_dev

namespace huv {

namespace {

// Rows of disjoint x runs for every clip (host, FP64).
void decompose(const huv_rect_clips& in, int n_clips, double L, std::vector<int32_t>& clip_rows,
               std::vector<huv_dev::RectRowDev>& rows, std::vector<double2>& runs) {
  const double half = L / 2.0;
  clip_rows.assign(1, 0);
  for (int c = 0; c < n_clips; ++c) {
    const int b = in.offsets[c], e = in.offsets[c + 1];
    struct R {
      double x0, x1, y0, y1;
    };
    std::vector<R> rs;
    std::vector<double> xe, ye;
    for (int i = b; i < e; ++i) {
      const huv_rect& q = in.rects[i];
      const double x0 = std::max(q.x - q.w / 2.0, -half), x1 = std::min(q.x + q.w / 2.0, half);
      const double y0 = std::max(q.y - q.h / 2.0, -half), y1 = std::min(q.y + q.h / 2.0, half);
      if (!(x1 > x0) || !(y1 > y0)) continue;
      rs.push_back(R{x0, x1, y0, y1});
      xe.push_back(x0);
      xe.push_back(x1);
      ye.push_back(y0);
      ye.push_back(y1);
    }
    std::sort(xe.begin(), xe.end());
    xe.erase(std::unique(xe.begin(), xe.end()), xe.end());
    std::sort(ye.begin(), ye.end());
    ye.erase(std::unique(ye.begin(), ye.end()), ye.end());
    const int E = static_cast<int>(xe.size());
    std::vector<int> cover(std::max(E - 1, 0));
    std::vector<double2> prev;
    for (size_t f = 0; f + 1 < ye.size(); ++f) {
      const double ya = ye[f], yb = ye[f + 1];
      std::fill(cover.begin(), cover.end(), 0);
      for (const R& r : rs)
        if (r.y0 <= ya && r.y1 >= yb) {
          const int e0 = static_cast<int>(std::lower_bound(xe.begin(), xe.end(), r.x0) - xe.begin());
          const int e1 = static_cast<int>(std::lower_bound(xe.begin(), xe.end(), r.x1) - xe.begin());
          for (int q = e0; q < e1; ++q) cover[q] = 1;
        }
      std::vector<double2> row;
      for (int q = 0; q + 1 < E;) {
        if (!cover[q]) {
          ++q;
          continue;
        }
        int q1 = q;
        while (q1 + 1 < E && cover[q1]) ++q1;
        row.push_back(make_double2(xe[q], xe[q1]));
        q = q1;
      }
      const bool same = !rows.empty() && static_cast<int>(rows.size()) > clip_rows.back() && row.size() == prev.size() &&
                        rows.back().y1 == ya &&
                        std::equal(row.begin(), row.end(), prev.begin(),
                                   [](const double2& u, const double2& v) { return u.x == v.x && u.y == v.y; });
      if (row.empty()) {
        prev.clear();
        continue;
      }
      if (same) {
        rows.back().y1 = yb;
      } else {
        huv_dev::RectRowDev rr{ya, yb, static_cast<int32_t>(runs.size()), static_cast<int32_t>(row.size())};
        rows.push_back(rr);
        runs.insert(runs.end(), row.begin(), row.end());
      }
      prev = row;
    }
    clip_rows.push_back(static_cast<int32_t>(rows.size()));
  }
}

}  // namespace

void Engine::check_rects(const huv_batch& b) const {
  const auto* in = static_cast<const huv_rect_clips*>(b.input);
  if (!in || !in->offsets || (in->offsets[b.n_clips] > in->offsets[0] && !in->rects))
    throw Error(HUV_ERR_INVALID_PARAMETER, "rect clips: null pointer");
  if (in->offsets[0] < 0) throw Error(HUV_ERR_INVALID_PARAMETER, "rect clips: offsets must be >= 0");
  for (int c = 0; c < b.n_clips; ++c)
    if (in->offsets[c + 1] < in->offsets[c]) throw Error(HUV_ERR_INVALID_PARAMETER, "rect clips: offsets decrease");
  for (int i = in->offsets[0]; i < in->offsets[b.n_clips]; ++i) {
    const huv_rect& q = in->rects[i];
    if (!(std::isfinite(q.x) && std::isfinite(q.y) && std::isfinite(q.w) && std::isfinite(q.h)) || q.w < 0 ||
        q.h < 0)
      throw Error(HUV_ERR_INVALID_PARAMETER, "rect clips: coordinates must be finite, sizes >= 0");
  }
  if (!(std::isfinite(in->feature_re) && std::isfinite(in->feature_im) && std::isfinite(in->background_re) &&
        std::isfinite(in->background_im)))
    throw Error(HUV_ERR_INVALID_PARAMETER, "rect clips: amplitudes must be finite");
}

void Engine::upload_rects(const huv_batch& b, int hb, cudaStream_t st) {
  const auto* in = static_cast<const huv_rect_clips*>(b.input);
  rect.dv = make_double2(in->feature_re - in->background_re, in->feature_im - in->background_im);
  rect.bg = make_double2(in->background_re, in->background_im);
  auto grow = [](void*& p, size_t& cap, size_t bytes) {
    if (bytes <= cap) return;
    if (p) cudaFree(p);
    p = nullptr;
    cap = 0;
    check_cuda(cudaMalloc(&p, bytes), "cudaMalloc(rect table)");
    cap = bytes;
  };
  cudaStreamCaptureStatus capture = cudaStreamCaptureStatusNone;
  check_cuda(cudaStreamIsCapturing(st, &capture), "cudaStreamIsCapturing");
  // Clips that fit rect_sort's shared memory are resolved on the device, as
  // long as the batch's tables (X, Y and both edge tables: 128 bytes per
  // rectangle and order) stay moderate; the copies are ordered on the stream.
  const int total = in->offsets[b.n_clips] - in->offsets[0];
  int most = 0;
  for (int c = 0; c < b.n_clips; ++c) most = std::max(most, in->offsets[c + 1] - in->offsets[c]);
  const int B = 2 * hb + 1;
  rect.on_device = most <= huv_dev::kRectSortMax && b.n_clips <= 65535 && B <= 255 &&
                   static_cast<size_t>(total) * B * 128 <= size_t(512) << 20;
  if (rect.on_device) {
    rect.most = most;
    rect.total = total;
    rect.clips = b.n_clips;
    // One copy of [rectangles][offsets], from pageable memory of our own: it
    // is staged before the call returns, whatever memory the caller's arrays
    // are in.
    const size_t rb = sizeof(huv_rect) * total, ob = sizeof(int32_t) * (b.n_clips + 1);
    rect.stage.resize(rb + ob);
    if (total > 0) std::memcpy(rect.stage.data(), in->rects + in->offsets[0], rb);
    std::memcpy(rect.stage.data() + rb, in->offsets, ob);
    grow(rect.dev, rect.dev_cap, rb + ob);
    // Inside a stream capture an asynchronous copy would become a node that
    // reads `stage` at every launch of the graph, when the vector may long have
    // moved.  The synchronous copy is made there and then, as the copies of the
    // host-resolved tables are.
    check_cuda(capture == cudaStreamCaptureStatusNone
                   ? cudaMemcpyAsync(rect.dev, rect.stage.data(), rb + ob, cudaMemcpyHostToDevice, st)
                   : cudaMemcpy(rect.dev, rect.stage.data(), rb + ob, cudaMemcpyHostToDevice),
               "upload rects");
    return;
  }
  std::vector<int32_t> clip_rows;
  std::vector<huv_dev::RectRowDev> rows;
  std::vector<double2> runs;
  decompose(*in, b.n_clips, n * pixel_nm, clip_rows, rows, runs);
  rect.n_rows = static_cast<int>(rows.size());
  grow(rect.clip_rows, rect.clip_rows_cap, sizeof(int32_t) * clip_rows.size());
  grow(rect.rows, rect.rows_cap, sizeof(huv_dev::RectRowDev) * std::max<size_t>(rows.size(), 1));
  grow(rect.runs, rect.runs_cap, sizeof(double2) * std::max<size_t>(runs.size(), 1));
  auto copy = [&](void* dst, const void* src, size_t bytes) {
    if (capture == cudaStreamCaptureStatusNone)
      upload(dst, src, bytes, "upload rect table");
    else  // no synchronisation inside a capture
      check_cuda(cudaMemcpy(dst, src, bytes, cudaMemcpyHostToDevice), "upload rect table");
  };
  copy(rect.clip_rows, clip_rows.data(), sizeof(int32_t) * clip_rows.size());
  if (!rows.empty()) {
    copy(rect.rows, rows.data(), sizeof(huv_dev::RectRowDev) * rows.size());
    copy(rect.runs, runs.data(), sizeof(double2) * runs.size());
  }
}

void Engine::rect_band(int c0, int nc, int hb, const float* W, float2* Mband, float* mean, cudaStream_t st) {
  const int B = 2 * hb + 1;
  if (B > 255) throw Error(HUV_ERR_UNSUPPORTED, "rect clips: band wider than 255 orders");
  const double L = n * pixel_nm;
  // Coefficients of every row of the batch (rows of later chunks are cheap
  // to recompute; the table is per batch).
  const size_t n_rows = static_cast<size_t>(std::max(rect.on_device ? 2 * rect.total : rect.n_rows, 1));
  const size_t n_edges = rect.on_device ? 2 * n_rows : 0;  // x edges, y edges
  const size_t tab = rect.on_device ? sizeof(double4) * n_rows / 2 + sizeof(double) * n_rows + sizeof(int2) * rect.clips + 64 : 0;
  const size_t need = sizeof(double2) * (2 * n_rows + n_edges) * B + tab;
  if (need > rect.coef_cap) {
    if (rect.coef) cudaFree(rect.coef);
    rect.coef = nullptr;
    rect.coef_cap = 0;
    check_cuda(cudaMalloc(&rect.coef, need), "cudaMalloc(rect coefficients)");
    rect.coef_cap = need;
  }
  double2* X = static_cast<double2*>(rect.coef);
  double2* Y = X + n_rows * B;
  double2 *EX = Y + n_rows * B, *EY = EX + n_rows * B;
  double4* sorted = reinterpret_cast<double4*>((reinterpret_cast<uintptr_t>(EX + n_edges * B) + 31) & ~uintptr_t(31));
  double* ys = reinterpret_cast<double*>(sorted + (n_rows + 1) / 2);
  int2* counts = reinterpret_cast<int2*>(ys + n_rows);
  const int32_t* offs = rect.on_device ? reinterpret_cast<const int32_t*>(static_cast<const huv_rect*>(rect.dev) + rect.total)
                                       : static_cast<const int32_t*>(rect.clip_rows);
  if (rect.on_device) {
    if (c0 == 0) {
      int cap = 1;
      while (cap < rect.most) cap <<= 1;
      huv_dev::rect_sort<<<rect.clips, 256, cap * (2 * sizeof(double) + sizeof(int16_t)), st>>>(
          static_cast<const double*>(rect.dev), offs, rect.total, L / 2.0, cap, sorted, ys, counts);
      const int vals = 4 * std::max(rect.most, 1) * B, rows = 2 * std::max(rect.most, 1);
      huv_dev::rect_edges<<<dim3(std::min((vals + 255) / 256, 64), rect.clips), 256, 0, st>>>(offs, rect.total, counts, sorted, ys, hb,
                                                                                             L, EX, EY);
      huv_dev::rect_rows<<<dim3(std::min((rows + 7) / 8, 64), rect.clips), 256, 0, st>>>(offs, rect.total, counts, sorted, ys, EX, EY,
                                                                                        hb, X, Y);
      check_cuda(cudaGetLastError(), "rect_rows");
    }
  } else if (c0 == 0 && rect.n_rows > 0) {
    const int threads = 256, warps = threads / 32;
    huv_dev::rect_row_coef<<<(rect.n_rows + warps - 1) / warps, threads, 0, st>>>(
        static_cast<const huv_dev::RectRowDev*>(rect.rows), static_cast<const double2*>(rect.runs), rect.n_rows, hb,
        L, X, Y);
    check_cuda(cudaGetLastError(), "rect_row_coef");
  }
  const int tiles = (B + huv_dev::kRectTY - 1) / huv_dev::kRectTY;
  float* parts = (W && mean) ? mean + nc : nullptr;
  const double n2 = static_cast<double>(n) * n;
  const size_t sm = sizeof(double2) * 16 * (huv_dev::kRectTY + B);
  huv_dev::rect_band_gemm<<<dim3(tiles, nc), 256, sm, st>>>(
      offs, rect.total, rect.on_device ? counts : nullptr, X, Y, c0, hb, n, rect.dv,
      make_double2(rect.bg.x * n2, rect.bg.y * n2), W, Mband, parts);
  check_cuda(cudaGetLastError(), "rect_band_gemm");
  if (parts) {
    huv_dev::rect_mean_reduce<<<(nc + 127) / 128, 128, 0, st>>>(parts, tiles, nc, mean);
    check_cuda(cudaGetLastError(), "mean_reduce(rects)");
  }
}

}  // namespace huv
