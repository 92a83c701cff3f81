// Field pass of narrow bands: evaluation grids M = 16 R, R = 1 .. 6, M > 4h.
//
// One kernel does what the row and column kernels of the wider grids do in
// two: for every SOCS kernel k the band product kappa_k . M, the zero-padded
// inverse FFT along x and along y, and sum_k |E_k|^2 in registers, then
// normalisation, flare and the FP16 hi/lo planes of I_M / interp_scale(mean)
// that the separable interpolation reads.  The row transforms stay in shared
// memory.  A block takes KB kernels at a time, so that the first column pass
// (one radix-16 butterfly per thread) fills its T = KB M^2 / 16 threads, and
// the kernels of one image are split over a cluster of blocks whose partial
// sums are added through distributed shared memory in a fixed order.  The
// flare mean sum_f W(f) |M(f)|^2 is summed here as well, and one launch takes
// several focus planes of the same clips (blockIdx.z).
//
// What bounds it: for one image the latency of a block's chain (four barriers
// per KB kernels), which is why the kernels are spread over the cluster; for a
// batch instruction issue.  The radix-4 pair it replaces ran all K kernels of
// a strip of columns in one block (36 of 70 us of a 256^2 image at M = 64),
// on power-of-two grids only (M = 128 where 80 or 96 suffice), and its images
// went through the band transform to the output grid.  Whole calls, before and
// after: one 256^2 EUV clip 70 -> 31 us, 7 complex 512^2 ArF clips 92 -> 38 us,
// one clip at 21 planes of focus (189 launches before, 5 now) 1,352 -> 39 us.
#include <cooperative_groups.h>
#include <cuda_fp16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include <algorithm>

#include "../engine.hpp"
#include "fft_reg.cuh"

namespace huv_dev {

namespace cgx = cooperative_groups;

constexpr int kSmallPlanes = 16;   // focus planes per launch
constexpr int kSmallMaxSplit = 8;  // blocks of one image (a portable cluster)

struct SmallPlanes {
  const float2* kband[kSmallPlanes];
  const float* W[kSmallPlanes];
  int K[kSmallPlanes];
  float keep[kSmallPlanes], flare[kSmallPlanes];
};

__host__ __device__ constexpr int fs_kb(int M) { return M == 16 ? 16 : M == 32 ? 4 : M == 48 ? 2 : 1; }
__host__ __device__ constexpr int fs_work(int M) { return fs_kb(M) * M * M / 16; }          // butterflies of a column pass
__host__ __device__ constexpr int fs_threads(int M) { return (fs_work(M) + 31) / 32 * 32; }
// float2 elements: column buffer (row buffer and partial sums alias it), row
// transforms, band products' factors, twiddles
__host__ __device__ constexpr size_t fs_smem(int M, int B) {
  return sizeof(float2) * (static_cast<size_t>(fs_kb(M)) * M * M + static_cast<size_t>(fs_kb(M)) * M * B +
                           static_cast<size_t>(fs_kb(M) + 1) * B * B + M);
}
// Blocks per image: about three rounds of KB of the set's K kernels each, at
// most a portable cluster.  A function of K and M alone, so that an image does
// not depend on the batch it is in; real masks keep it for half the kernels,
// so that the planes of a focus sweep, of which the one in focus folds, share
// a launch.
__host__ __device__ inline int fs_split(int M, int K) {
  const int rounds = (K + fs_kb(M) - 1) / fs_kb(M);
  const int s = (rounds + 2) / 3;
  return s < 1 ? 1 : (s > kSmallMaxSplit ? kSmallMaxSplit : s);
}

// First pass (radix 16) of a zero-padded band of half-width h < M / 4 for
// butterfly j: `at(m)` gives the value at band index m = order + h.
template <int R, typename F>
__device__ __forceinline__ void fs_band16(int j, int h, float2 (&v)[16], F at) {
#pragma unroll
  for (int r = 0; r < 16; ++r) {
    if (r >= 4 && r < 12) continue;  // outside the band
    const int i = j + r * R;
    const int m = r < 4 ? (i <= h ? i + h : -1) : (i >= 16 * R - h ? i - 16 * R + h : -1);
    v[r] = m >= 0 ? at(m) : make_float2(0.f, 0.f);
  }
  fr_dft16_band<+1>(v);
}

template <int M>
__global__ void __launch_bounds__(fs_threads(M))
    socs_field_small(const __grid_constant__ SmallPlanes pl, const float2* __restrict__ Mband, int hb, int clips,
                     const float2* __restrict__ tw, float* __restrict__ mean, __half* __restrict__ split) {
  constexpr int R = M / 16, KB = fs_kb(M), T = fs_work(M), NT = fs_threads(M);
  constexpr int SR = KB * M / 2, SC = KB * M;           // row and column sequences
  constexpr int NR = R > 1 ? (16 * SR + T - 1) / T : 1;  // last-pass butterflies per thread, rows
  constexpr int NC = R > 1 ? (16 * SC + T - 1) / T : 1;  // and columns
  extern __shared__ float2 smem[];
  __shared__ float red[NT / 32];
  __shared__ float s_mean;
  const int t = threadIdx.x, B = 2 * hb + 1, BB = B * B;
  const int ks = blockIdx.x, nsplit = gridDim.x, clip = blockIdx.y, plane = blockIdx.z;
  float2* buf = smem;               // [M][SC], rows [M][SR]
  float2* rows = buf + KB * M * M;  // [SC][B]: x-major row transforms
  float2* sM = rows + KB * M * B;   // [B][B] mask band
  float2* sU = sM + BB;             // [KB][B][B] kernels of this round
  float2* sw = sU + KB * BB;        // [M] exp(+2 pi i t / M)
  const float2* kband = pl.kband[plane];
  const int K = pl.K[plane];
  const int k0 = K * ks / nsplit, k1 = K * (ks + 1) / nsplit;
  auto fetch = [&](int k) {
    const int n = min(KB, k1 - k) * BB;
    const float2* src = kband + static_cast<size_t>(k) * BB;
    for (int e = t; e < n; e += NT) fr_cp_async8(sU + e, src + e);
    fr_cp_commit();
  };
  fetch(k0);
  {
    // mask band, twiddles and the flare mean (every block of the cluster: its
    // blocks need no exchange before the last)
    const float2* Mc = Mband + static_cast<size_t>(clip) * BB;
    const float* W = pl.W[plane];
    float part = 0.f;
    for (int e = t; e < BB; e += NT) {
      const float2 v = Mc[e];
      sM[e] = v;
      part += W[e] * (v.x * v.x + v.y * v.y);
    }
    for (int e = t; e < M; e += NT) {
      const float2 w = tw[e];
      sw[e] = make_float2(w.x, -w.y);
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) part += __shfl_xor_sync(0xffffffffu, part, o);
    if ((t & 31) == 0) red[t >> 5] = part;
  }
  float acc[NC][R > 1 ? R : 16];
#pragma unroll
  for (int c = 0; c < NC; ++c)
#pragma unroll
    for (int p = 0; p < (R > 1 ? R : 16); ++p) acc[c][p] = 0.f;

  for (int k = k0; k < k1; k += KB) {
    fr_cp_wait<0>();
    __syncthreads();
    if (k == k0 && t == 0) {
      float s = 0.f;
      for (int w = 0; w < NT / 32; ++w) s += red[w];
      s_mean = s;
      if (ks == 0) mean[plane * clips + clip] = s;
    }
    // rows: first pass on the band products
    if (t < T / 2) {
      const int s = t % SR, j = t / SR, kk = s / (M / 2), my = s % (M / 2);
      float2 v[16];
      if (my < B && k + kk < k1) {
        const float2 *u = sU + kk * BB + my * B, *m = sM + my * B;
        fs_band16<R>(j, hb, v, [&](int q) { return fr_mul(u[q], m[q]); });
      } else {
#pragma unroll
        for (int r = 0; r < 16; ++r) v[r] = make_float2(0.f, 0.f);
      }
      if constexpr (R > 1) {
#pragma unroll
        for (int r = 0; r < 16; ++r) buf[(j * 16 + r) * SR + s] = v[r];
      } else if (my < B) {
#pragma unroll
        for (int r = 0; r < 16; ++r) rows[(kk * M + r) * B + my] = v[r];
      }
    }
    __syncthreads();
    if (k + KB < k1) fetch(k + KB);  // sU is free: the first pass was its last reader
    if constexpr (R > 1) {
#pragma unroll
      for (int c = 0; c < NR; ++c) {
        const int u = t + c * T;
        if (t >= T || u >= 16 * SR) break;
        const int s = u % SR, j = u / SR, kk = s / (M / 2), my = s % (M / 2);
        float2 v[R];
#pragma unroll
        for (int r = 0; r < R; ++r) v[r] = buf[(j + r * 16) * SR + s];
#pragma unroll
        for (int r = 1; r < R; ++r) v[r] = fr_mul(v[r], sw[r * j]);
        fr_dft<R, +1>(v);
        if (my < B)
#pragma unroll
          for (int p = 0; p < R; ++p) rows[(kk * M + j + p * 16) * B + my] = v[p];
      }
      __syncthreads();
    }
    // columns
    if (t < T) {
      const int s = t % SC, j = t / SC;
      const float2* col = rows + s * B;
      float2 v[16];
      fs_band16<R>(j, hb, v, [&](int q) { return col[q]; });
      if constexpr (R > 1) {
#pragma unroll
        for (int r = 0; r < 16; ++r) buf[(j * 16 + r) * SC + s] = v[r];
      } else {
#pragma unroll
        for (int r = 0; r < 16; ++r) acc[0][r] += v[r].x * v[r].x + v[r].y * v[r].y;
      }
    }
    if constexpr (R > 1) {
      __syncthreads();
#pragma unroll
      for (int c = 0; c < NC; ++c) {
        const int u = t + c * T;
        if (t >= T || u >= 16 * SC) break;
        const int s = u % SC, j = u / SC;
        float2 v[R];
#pragma unroll
        for (int r = 0; r < R; ++r) v[r] = buf[(j + r * 16) * SC + s];
#pragma unroll
        for (int r = 1; r < R; ++r) v[r] = fr_mul(v[r], sw[r * j]);
        fr_dft<R, +1>(v);
#pragma unroll
        for (int p = 0; p < R; ++p) acc[c][p] += v[p].x * v[p].x + v[p].y * v[p].y;
      }
    }
    // No barrier here: the next round's first writes (buf by its row pass)
    // come after its loop-top barrier.
  }
  // partial sums [kk][y][x] over buf, then the cluster's in order
  __syncthreads();
  float* part = reinterpret_cast<float*>(buf);
  if constexpr (R > 1) {
#pragma unroll
    for (int c = 0; c < NC; ++c) {
      const int u = t + c * T;
      if (t >= T || u >= 16 * SC) break;
      const int s = u % SC, j = u / SC;
#pragma unroll
      for (int p = 0; p < R; ++p) part[(s / M * M + j + p * 16) * M + s % M] = acc[c][p];
    }
  } else if (t < T) {
#pragma unroll
    for (int r = 0; r < 16; ++r) part[(t / M * M + r) * M + t % M] = acc[0][r];
  }
  cgx::cluster_group cl = cgx::this_cluster();
  cl.sync();
  const float mn = s_mean, add = pl.flare[plane] * mn, keep = pl.keep[plane], inv = 1.f / interp_scale(mn);
  __half2* out = reinterpret_cast<__half2*>(split + static_cast<size_t>(plane * clips + clip) * 2 * M * M);
  for (int e = ks * NT + t; e < M * M / 2; e += nsplit * NT) {
    float2 s = make_float2(0.f, 0.f);
    for (int q = 0; q < nsplit; ++q) {
      const float2* src = reinterpret_cast<const float2*>(cl.map_shared_rank(part, q)) + e;
#pragma unroll 4
      for (int kk = 0; kk < KB; ++kk) {
        const float2 v = src[kk * (M * M / 2)];
        s.x += v.x;
        s.y += v.y;
      }
    }
    const float a = (keep * s.x + add) * inv, b = (keep * s.y + add) * inv;
    const __half2 hi = __floats2half2_rn(a, b);
    const float2 hf = __half22float2(hi);
    out[e] = hi;
    out[M * M / 2 + e] = __floats2half2_rn(a - hf.x, b - hf.y);
  }
  cl.sync();  // no block leaves while another reads its partial sums
}

// Adjoint of the field pass on the same grids: Q = sum_k conj(kappa_k) .
// band(FFT(G0 . E_k)), G0 = keep G + flare_over_n sums[mask][1].  The fields
// E_k are made again from the mask band (as socs_field_small makes them),
// multiplied by G0 at each thread's own points, transformed back along y and x
// within the band, and conj(kappa_k) times the result is summed in registers
// over the block's kernels, then over the cluster in order.  Nothing but Q is
// written: the two radix-4 kernels it replaces kept every field's transform in
// memory and ran all kernels of a strip in one block (3 masks of 256^2, M =
// 64, 20 kernels: 69 -> 13 us).
// grid: (split, masks), clusters of split.
template <int M>
__global__ void __launch_bounds__(fs_threads(M))
    ilt_adj_small(const float2* __restrict__ kband, const float2* __restrict__ Mband, const float* __restrict__ G, int K,
                  int hb, float keep, const double* __restrict__ sums, float flare_over_n,
                  const float2* __restrict__ tw, float2* __restrict__ Q) {
  constexpr int R = M / 16, KB = fs_kb(M), T = fs_work(M), NT = fs_threads(M);
  constexpr int SR = KB * M / 2, SC = KB * M;
  constexpr int NR = R > 1 ? (16 * SR + T - 1) / T : 1;
  constexpr int NC = R > 1 ? (16 * SC + T - 1) / T : 1;
  constexpr int RO = R > 1 ? R : 16;  // outputs of one butterfly of the last pass
  extern __shared__ float2 smem[];
  const int t = threadIdx.x, B = 2 * hb + 1, BB = B * B;
  const int ks = blockIdx.x, nsplit = gridDim.x, mask = blockIdx.y;
  float2* buf = smem;               // [M][SC], rows [M][SR]
  float2* rows = buf + KB * M * M;  // [SC][B]
  float2* sM = rows + KB * M * B;   // [B][B]
  float2* sU = sM + BB;             // [2][KB][B][B]
  float2* sw = sU + 2 * KB * BB;    // [M] exp(+2 pi i t / M)
  const int k0 = K * ks / nsplit, k1 = K * (ks + 1) / nsplit;
  auto fetch = [&](int k) {
    const int n = min(KB, k1 - k) * BB;
    const float2* src = kband + static_cast<size_t>(k) * BB;
    float2* dst = sU + (((k - k0) / KB) & 1) * KB * BB;
    for (int e = t; e < n; e += NT) fr_cp_async8(dst + e, src + e);
    fr_cp_commit();
  };
  fetch(k0);
  for (int e = t; e < BB; e += NT) sM[e] = Mband[static_cast<size_t>(mask) * BB + e];
  for (int e = t; e < M; e += NT) {
    const float2 w = tw[e];
    sw[e] = make_float2(w.x, -w.y);
  }
  // G0 at the thread's points of the last inverse pass
  const float add = flare_over_n * static_cast<float>(sums[mask * 2 + 1]);
  const float* Gm = G + static_cast<size_t>(mask) * M * M;
  float g[NC][RO];
#pragma unroll
  for (int c = 0; c < NC; ++c) {
    const int u = R > 1 ? t + c * T : t;
    const int x = (u % SC) % M, j = R > 1 ? (u / SC) % 16 : 0;  // guarded butterflies read a valid point
#pragma unroll
    for (int p = 0; p < RO; ++p) g[c][p] = keep * Gm[(R > 1 ? j + p * 16 : p) * M + x] + add;
  }
  float2 acc[NR][RO];
#pragma unroll
  for (int c = 0; c < NR; ++c)
#pragma unroll
    for (int p = 0; p < RO; ++p) acc[c][p] = make_float2(0.f, 0.f);
  auto band = [&](int i) { return i <= hb ? i + hb : (i >= M - hb ? i - M + hb : -1); };

  for (int k = k0; k < k1; k += KB) {
    const float2* U = sU + (((k - k0) / KB) & 1) * KB * BB;
    fr_cp_wait<0>();
    __syncthreads();
    if (k + KB < k1) fetch(k + KB);  // the other buffer: its last readers passed the barrier above
    // ---- fields, as in socs_field_small
    if (t < T / 2) {
      const int s = t % SR, j = t / SR, kk = s / (M / 2), my = s % (M / 2);
      float2 v[16];
      if (my < B && k + kk < k1) {
        const float2 *u = U + kk * BB + my * B, *m = sM + my * B;
        fs_band16<R>(j, hb, v, [&](int q) { return fr_mul(u[q], m[q]); });
      } else {
#pragma unroll
        for (int r = 0; r < 16; ++r) v[r] = make_float2(0.f, 0.f);
      }
      if constexpr (R > 1) {
#pragma unroll
        for (int r = 0; r < 16; ++r) buf[(j * 16 + r) * SR + s] = v[r];
      } else if (my < B) {
#pragma unroll
        for (int r = 0; r < 16; ++r) rows[(kk * M + r) * B + my] = v[r];
      }
    }
    __syncthreads();
    if constexpr (R > 1) {
#pragma unroll
      for (int c = 0; c < NR; ++c) {
        const int u = t + c * T;
        if (t >= T || u >= 16 * SR) break;
        const int s = u % SR, j = u / SR, kk = s / (M / 2), my = s % (M / 2);
        float2 v[R];
#pragma unroll
        for (int r = 0; r < R; ++r) v[r] = buf[(j + r * 16) * SR + s];
#pragma unroll
        for (int r = 1; r < R; ++r) v[r] = fr_mul(v[r], sw[r * j]);
        fr_dft<R, +1>(v);
        if (my < B)
#pragma unroll
          for (int p = 0; p < R; ++p) rows[(kk * M + j + p * 16) * B + my] = v[p];
      }
      __syncthreads();
    }
    float2 f[16];  // a column butterfly
    if (t < T) {
      const int s = t % SC, j = t / SC;
      const float2* col = rows + s * B;
      fs_band16<R>(j, hb, f, [&](int q) { return col[q]; });
      if constexpr (R > 1) {
#pragma unroll
        for (int r = 0; r < 16; ++r) buf[(j * 16 + r) * SC + s] = f[r];
      } else {
#pragma unroll
        for (int r = 0; r < 16; ++r) f[r] = make_float2(f[r].x * g[0][r], f[r].y * g[0][r]);
      }
    }
    __syncthreads();
    // ---- times G0 (in place: a butterfly reads and writes the points j + 16 r), and back along y
    if constexpr (R > 1) {
#pragma unroll
      for (int c = 0; c < NC; ++c) {
        const int u = t + c * T;
        if (t >= T || u >= 16 * SC) break;
        const int s = u % SC, j = u / SC;
        float2 v[R];
#pragma unroll
        for (int r = 0; r < R; ++r) v[r] = buf[(j + r * 16) * SC + s];
#pragma unroll
        for (int r = 1; r < R; ++r) v[r] = fr_mul(v[r], sw[r * j]);
        fr_dft<R, +1>(v);
#pragma unroll
        for (int p = 0; p < R; ++p) buf[(j + p * 16) * SC + s] = make_float2(v[p].x * g[c][p], v[p].y * g[c][p]);
      }
      __syncthreads();
      if (t < T) {
        const int s = t % SC, j = t / SC;
#pragma unroll
        for (int r = 0; r < 16; ++r) f[r] = buf[(j + r * R) * SC + s];
      }
      __syncthreads();
    }
    if (t < T) {
      const int s = t % SC, j = t / SC;
      fr_dft<16, -1>(f);
      if constexpr (R > 1) {
#pragma unroll
        for (int r = 0; r < 16; ++r) buf[(j * 16 + r) * SC + s] = f[r];
      } else {
#pragma unroll
        for (int r = 0; r < 16; ++r)
          if (band(r) >= 0) rows[s * B + band(r)] = f[r];
      }
    }
    __syncthreads();
    if constexpr (R > 1) {
#pragma unroll
      for (int c = 0; c < NC; ++c) {
        const int u = t + c * T;
        if (t >= T || u >= 16 * SC) break;
        const int s = u % SC, j = u / SC;
        float2 v[R];
#pragma unroll
        for (int r = 0; r < R; ++r) v[r] = buf[(j + r * 16) * SC + s];
#pragma unroll
        for (int r = 1; r < R; ++r) v[r] = fr_mul(v[r], make_float2(sw[r * j].x, -sw[r * j].y));
        fr_dft<R, -1>(v);
#pragma unroll
        for (int p = 0; p < R; ++p) {
          const int m = band(j + p * 16);
          if (m >= 0) rows[s * B + m] = v[p];
        }
      }
      __syncthreads();
    }
    // ---- back along x, times conj(kappa)
    if (t < T / 2) {
      const int s = t % SR, j = t / SR, kk = s / (M / 2), my = s % (M / 2);
      float2 v[16];
#pragma unroll
      for (int r = 0; r < 16; ++r) v[r] = my < B ? rows[(kk * M + j + r * R) * B + my] : make_float2(0.f, 0.f);
      fr_dft<16, -1>(v);
      if constexpr (R > 1) {
#pragma unroll
        for (int r = 0; r < 16; ++r) buf[(j * 16 + r) * SR + s] = v[r];
      } else if (my < B && k + kk < k1) {
#pragma unroll
        for (int r = 0; r < 16; ++r)
          if (band(r) >= 0) {
            const float2 u = U[kk * BB + my * B + band(r)];
            acc[0][r].x += u.x * v[r].x + u.y * v[r].y;
            acc[0][r].y += u.x * v[r].y - u.y * v[r].x;
          }
      }
    }
    if constexpr (R > 1) {
      __syncthreads();
#pragma unroll
      for (int c = 0; c < NR; ++c) {
        const int u = t + c * T;
        if (t >= T || u >= 16 * SR) break;
        const int s = u % SR, j = u / SR, kk = s / (M / 2), my = s % (M / 2);
        float2 v[R];
#pragma unroll
        for (int r = 0; r < R; ++r) v[r] = buf[(j + r * 16) * SR + s];
#pragma unroll
        for (int r = 1; r < R; ++r) v[r] = fr_mul(v[r], make_float2(sw[r * j].x, -sw[r * j].y));
        fr_dft<R, -1>(v);
        if (my < B && k + kk < k1)
#pragma unroll
          for (int p = 0; p < R; ++p) {
            const int m = band(j + p * 16);
            if (m >= 0) {
              const float2 q = U[kk * BB + my * B + m];
              acc[c][p].x += q.x * v[p].x + q.y * v[p].y;
              acc[c][p].y += q.x * v[p].y - q.y * v[p].x;
            }
          }
      }
    }
  }
  // partial sums [kk][my][mx] over buf, then the cluster's in order
  __syncthreads();
#pragma unroll
  for (int c = 0; c < NR; ++c) {
    const int u = R > 1 ? t + c * T : t;
    if (R > 1 ? (t >= T || u >= 16 * SR) : t >= T / 2) break;
    const int s = u % SR, j = u / SR, kk = s / (M / 2), my = s % (M / 2);
    if (my < B)
#pragma unroll
      for (int p = 0; p < RO; ++p) {
        const int m = band(R > 1 ? j + p * 16 : p);
        if (m >= 0) buf[kk * BB + my * B + m] = acc[c][p];
      }
  }
  cgx::cluster_group cl = cgx::this_cluster();
  cl.sync();
  for (int e = ks * NT + t; e < BB; e += nsplit * NT) {
    float2 s = make_float2(0.f, 0.f);
    for (int q = 0; q < nsplit; ++q) {
      const float2* src = cl.map_shared_rank(buf, q) + e;
      for (int kk = 0; kk < KB; ++kk) s = fr_add(s, src[kk * BB]);
    }
    Q[static_cast<size_t>(mask) * BB + e] = s;
  }
  cl.sync();  // no block leaves while another reads its partial sums
}

}  // namespace huv_dev

namespace huv_launch {

bool interp_fused_ok(int M, int n);

// Whether the narrow-band field kernel serves an M grid and band half-width hb.
bool field_small_ok(int M, int hb) { return M % 16 == 0 && M >= 16 && M <= 96 && 4 * hb < M; }

namespace {
template <int M>
cudaError_t launch_small(const huv_dev::SmallPlanes& pl, int planes, int split, const float2* Mband, int hb, int clips,
                         const float2* tw, float* mean, void* out, cudaStream_t st) {
  static std::atomic<uint64_t> attr{0};
  huv::once_per_device(attr, [] {
    huv::check_cuda(cudaFuncSetAttribute(huv_dev::socs_field_small<M>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         static_cast<int>(huv_dev::fs_smem(M, M / 2))),
                    "cudaFuncSetAttribute(field_small)");
  });
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(split, clips, planes);
  cfg.blockDim = dim3(huv_dev::fs_threads(M));
  cfg.dynamicSmemBytes = huv_dev::fs_smem(M, 2 * hb + 1);
  cfg.stream = st;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.x = split;
  at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, huv_dev::socs_field_small<M>, pl, Mband, hb, clips, tw, mean,
                            static_cast<__half*>(out));
}
template <int M>
cudaError_t launch_adj(const float2* kband, const float2* Mband, const float* G, int K, int hb, float keep,
                       const double* sums, float flare_over_n, int masks, const float2* tw, float2* Q, cudaStream_t st) {
  static std::atomic<uint64_t> attr{0};
  auto smem = [](int B) { return huv_dev::fs_smem(M, B) + sizeof(float2) * huv_dev::fs_kb(M) * B * B; };
  huv::once_per_device(attr, [&] {
    huv::check_cuda(cudaFuncSetAttribute(huv_dev::ilt_adj_small<M>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         static_cast<int>(smem(M / 2))),
                    "cudaFuncSetAttribute(ilt_adj_small)");
  });
  const int split = std::min(huv_dev::fs_split(M, K), K);
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(split, masks);
  cfg.blockDim = dim3(huv_dev::fs_threads(M));
  cfg.dynamicSmemBytes = smem(2 * hb + 1);
  cfg.stream = st;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.x = split;
  at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, huv_dev::ilt_adj_small<M>, kband, Mband, G, K, hb, keep, sums, flare_over_n, tw, Q);
}
}  // namespace

// Q of every mask on the power-of-two grids that the ILT uses below 128.
bool ilt_adj_small_ok(int M, int hb) { return (M == 16 || M == 32 || M == 64) && field_small_ok(M, hb); }
cudaError_t ilt_adj_small(const float2* kband, const float2* Mband, const float* G, int M, int K, int hb, float keep,
                          const double* sums, float flare_over_n, int masks, const float2* tw, float2* Q,
                          cudaStream_t st) {
  switch (M) {
    case 16: return launch_adj<16>(kband, Mband, G, K, hb, keep, sums, flare_over_n, masks, tw, Q, st);
    case 32: return launch_adj<32>(kband, Mband, G, K, hb, keep, sums, flare_over_n, masks, tw, Q, st);
    case 64: return launch_adj<64>(kband, Mband, G, K, hb, keep, sums, flare_over_n, masks, tw, Q, st);
    default: return cudaErrorInvalidValue;
  }
}

// I_M / interp_scale(mean) of every plane and clip as FP16 planes
// [plane][clip][2][M][M], and the flare means [plane][clip].  The planes' sets
// share hb; planes whose kernels split differently go in launches of their own.
cudaError_t field_small(const huv::SmallPlane* p, int planes, const float2* Mband, int M, int hb, int clips,
                        const float2* tw, float* mean, void* out, cudaStream_t st) {
  const size_t img = static_cast<size_t>(clips) * 2 * M * M;
  for (int a = 0; a < planes;) {
    const int split = p[a].split;
    huv_dev::SmallPlanes pl{};
    int c = 0;
    for (; a + c < planes && c < huv_dev::kSmallPlanes && p[a + c].split == split; ++c) {
      pl.kband[c] = p[a + c].kband;
      pl.W[c] = p[a + c].W;
      pl.K[c] = p[a + c].K;
      pl.keep[c] = p[a + c].keep;
      pl.flare[c] = p[a + c].flare;
    }
    float* mn = mean + static_cast<size_t>(a) * clips;
    void* o = static_cast<__half*>(out) + img * a;
    cudaError_t e;
    switch (M) {
      case 16: e = launch_small<16>(pl, c, split, Mband, hb, clips, tw, mn, o, st); break;
      case 32: e = launch_small<32>(pl, c, split, Mband, hb, clips, tw, mn, o, st); break;
      case 48: e = launch_small<48>(pl, c, split, Mband, hb, clips, tw, mn, o, st); break;
      case 64: e = launch_small<64>(pl, c, split, Mband, hb, clips, tw, mn, o, st); break;
      case 80: e = launch_small<80>(pl, c, split, Mband, hb, clips, tw, mn, o, st); break;
      case 96: e = launch_small<96>(pl, c, split, Mband, hb, clips, tw, mn, o, st); break;
      default: return cudaErrorInvalidValue;
    }
    if (e != cudaSuccess) return e;
    a += c;
  }
  return cudaGetLastError();
}

}  // namespace huv_launch

namespace huv {

int Engine::small_grid(const DeviceSet& ds, int requested) const {
  const int m = requested > 0 ? requested : 16 * (4 * ds.hb / 16 + 1);  // the smallest multiple of 16 above 4h
  return huv_launch::field_small_ok(m, ds.hb) && huv_launch::interp_fused_ok(m, n) && hybrid_supported(ds, 16) ? m : 0;
}

void Engine::run_small_form(const huv_batch& b, DeviceSet* const* sets, const int* K_use, const float* const* W_use,
                            int planes, int M, float* out, cudaStream_t st) {
  using namespace huv_launch;
  DeviceSet& ds = *sets[0];
  const int B = ds.B, hb = ds.hb;
  auto align = [](size_t v) { return (v + 255) & ~size_t(255); };
  const size_t in_elem = b.input_kind == HUV_INPUT_RASTER_U8
                             ? 1
                             : (b.input_kind == HUV_INPUT_RASTER_F32 ? 4 : (b.input_kind == HUV_INPUT_RECTS ? 0 : 8));
  const size_t npix = static_cast<size_t>(n) * n;
  const size_t per_x = align(sizeof(float2) * n * B), per_m = align(sizeof(float2) * B * B);
  const size_t per_i = align(sizeof(float) * M * M) * planes, per_mean = align(sizeof(float) * planes);
  const size_t per_clip = per_x + per_m + per_i + per_mean;
  // (grid dimensions y and z hold at most 65,535 problems)
  const int chunk = balanced_chunk(
      static_cast<int>(std::min<size_t>(std::max<size_t>(1, chunk_budget() / per_clip), std::max(1, 65535 / planes))),
      b.n_clips);
  char* base = static_cast<char*>(workspace(per_clip * chunk + 4096));
  float2* X = reinterpret_cast<float2*>(base);
  float2* Mb = reinterpret_cast<float2*>(base + per_x * chunk);
  void* IM = base + (per_x + per_m) * chunk;
  float* mean = reinterpret_cast<float*>(base + (per_x + per_m + per_i) * chunk);
  std::vector<SmallPlane> pl(planes);
  for (int p = 0; p < planes; ++p) {
    const int K = K_use && K_use[p] ? K_use[p] : sets[p]->K;
    const BandKernels bk = kernels_for(b, *sets[p], K, st);
    pl[p] = SmallPlane{bk.kband, W_use && W_use[p] ? W_use[p] : sets[p]->W, bk.K, std::min(huv_dev::fs_split(M, K), bk.K),
                       sets[p]->keep, sets[p]->flare};
  }
  int lgn = 0;
  while ((1 << lgn) < n) ++lgn;
  const float2* twn = twiddle_n(n);
  const float2* twm = twiddle_n(M);
  for (int c0 = 0; c0 < b.n_clips; c0 += chunk) {
    const int nc = std::min(chunk, b.n_clips - c0);
    const void* in = static_cast<const char*>(b.input) + in_elem * npix * c0;
    prof.begin("mask_band", st);
    if (b.input_kind == HUV_INPUT_RECTS)
      rect_band(c0, nc, hb, nullptr, Mb, nullptr, st);
    else
      check_cuda(band_forward(in, b.input_kind, n, lgn, hb, nc, X, Mb, b.pixel_transfer ? ds.ptx : nullptr, nullptr,
                              nullptr, twn, st, row_digit_table(hb), dev_err),
                 "band_forward");
    prof.end(st);
    prof.begin("socs_field_small", st);
    check_cuda(field_small(pl.data(), planes, Mb, M, hb, nc, twm, mean, IM, st), "socs_field_small");
    prof.end(st);
    prof.launches += 3 + (planes - 1) / huv_dev::kSmallPlanes;
    // the planes' images are contiguous when one chunk holds every clip
    if (nc == b.n_clips) {
      interp_separable(ds, M, planes * nc, IM, mean, nullptr, out, st, true);
      ++prof.launches;
    } else {
      for (int p = 0; p < planes; ++p)
        interp_separable(ds, M, nc, static_cast<char*>(IM) + sizeof(float) * M * M * nc * p, mean + static_cast<size_t>(nc) * p,
                         nullptr, out + npix * (static_cast<size_t>(p) * b.n_clips + c0), st, true);
      prof.launches += planes;
    }
  }
}

}  // namespace huv
