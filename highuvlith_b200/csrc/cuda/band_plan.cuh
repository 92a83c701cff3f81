// Columns per block of the band transform's column pass, and with it the room
// that the flare mean's partial sums need (csrc/cuda/socs_fft.cu): one rule for
// the launch and for everyone who sizes a workspace.
#pragma once
#include <cuda_runtime.h>

#include <algorithm>

#include "fft_block.cuh"
#include "fft_reg.cuh"

namespace huv_dev {

constexpr int kRectTY = 16;  // band rows per block of the rectangle spectrum (csrc/cuda/rects.cu)

// Whether the register-radix kernels (x-major band layout) apply to length L
// (128, 160, 192, 256, 512, 1024, 2048) and band half-width hb: every one of
// them within the shared-memory budget.
inline bool xt_fits(int L, int hb) {
  const int S = xt_S(L);
  if (S == 0 || 2 * hb >= L) return false;
  // the largest user: the column pass with two band buffers and two FFT buffers
  const size_t cols = 2 * static_cast<size_t>(S) * (2 * hb + 1) * sizeof(float2) +
                      2 * static_cast<size_t>(fr_buf(L, S)) * sizeof(float2);
  return cols <= static_cast<size_t>(kXtSmemMax);
}

// Band columns per block of the column pass on n points.
inline int band_cols_per_block(int n, int hb) {
  return xt_fits(n, hb) ? xt_S(n) : fit_units(4, 2 * sizeof(float2) * static_cast<size_t>(n));
}

// Partial sums of one clip's flare mean, at most: a block each, of the column
// pass over all 2 hb + 1 columns (half of them for real rasters) or of the
// rectangle spectrum.  Two columns per block at 2048 and 4096 points, one at
// 8192.
inline int band_mean_parts(int n, int hb) {
  const int B = 2 * hb + 1, u = std::min(band_cols_per_block(n, hb), kRectTY);
  return (B + u - 1) / u;
}

}  // namespace huv_dev
