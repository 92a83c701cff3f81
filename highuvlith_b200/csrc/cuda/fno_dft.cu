// DFTs of the FNO over its retained modes, and the lift.
//
// All of it is FP32 on CUDA cores.  Every sum keeps one fixed order of
// operations (given at each kernel): the results are rounded to BF16 before
// the channel GEMMs, where another order of the same FP32 sum flips enough
// roundings to show in the images (9e-4 of the largest pixel), so a kernel
// may change who adds but not in which order.
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include <algorithm>

#include "../engine.hpp"
#include "fft_reg.cuh"

namespace huv_dev {

namespace {
__device__ __forceinline__ void cp16(void* dst, const void* src) { fr_cp_async16(dst, src); }
__device__ __forceinline__ void load4(const __nv_bfloat16* p, float (&a)[4]) {
  const uint2 u = *reinterpret_cast<const uint2*>(p);
  a[0] = __uint_as_float(u.x << 16);
  a[1] = __uint_as_float(u.x & 0xffff0000u);
  a[2] = __uint_as_float(u.y << 16);
  a[3] = __uint_as_float(u.y & 0xffff0000u);
}
__device__ __forceinline__ void load4(const float* p, float (&a)[4]) {
  const float4 u = *reinterpret_cast<const float4*>(p);
  a[0] = u.x;
  a[1] = u.y;
  a[2] = u.z;
  a[3] = u.w;
}
// Two FP32 multiply-adds in one instruction (each rounded as fmaf).
__device__ __forceinline__ uint64_t pack2(float x, float y) {
  uint64_t r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(x), "f"(y));
  return r;
}
__device__ __forceinline__ float2 unpack2(uint64_t v) {
  float2 r;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(v));
  return r;
}
__device__ __forceinline__ void fma2(uint64_t& acc, uint64_t a, uint64_t b) {
  asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(acc) : "l"(a), "l"(b));
}
}  // namespace

// ------------------------------------------------------------ DFT along x
// out[r][kx][c] (complex) = sum_x in[r][x][c] e^{-2 pi i kx x / S}, rows r =
// (b, y), kx < m <= 16, C = 64; twt[x][16] holds the twiddles (zero past m).
// Order: x runs in chunks of min(128, S), each split over four thread groups
// (group g takes the g-th quarter of every chunk, in order, one fused
// multiply-add per term); the groups are added as ((0 + 1) + 2) + 3.
//
// 256 threads take two rows; a thread owns 8 kx x 4 c, so that a step of x
// costs five shared loads for 32 paired multiply-adds (bound by FP32 issue:
// the 4 x 4 tile it replaces spent five loads on 32 single ones and staged
// its input with blocking 2-byte loads).  Input and twiddles arrive by
// cp.async, two stages; a stage is a chunk of BF16 or half of one of FP32
// (the same bytes).  16 x 512^2 BF16: 1.21 -> 0.46 ms (0.57 with single
// multiply-adds); 8 x 512^2 FP32: 0.617 -> 0.26 ms.
constexpr int kDxRows = 2, kDxThreads = 128 * kDxRows;
template <typename T>
__host__ __device__ constexpr int dx_split() { return sizeof(T) == 4 ? 2 : 1; }  // stages per chunk
template <typename T>
__host__ __device__ constexpr size_t dx_stage_bytes() {
  return kDxRows * (128 / dx_split<T>()) * 64 * sizeof(T) + (128 / dx_split<T>()) * 16 * sizeof(float2);
}

template <typename T>
__global__ void __launch_bounds__(kDxThreads, 2) fno_dft_x(const T* __restrict__ in, int S, int m,
                                                     const float2* __restrict__ twt, float2* __restrict__ out,
                                                     int rows) {
  constexpr int C = 64;
  extern __shared__ __align__(128) uint8_t dsm8[];
  const int t = threadIdx.x;
  const int cg = t & 15, kg = (t >> 4) & 1, grp = (t >> 5) & 3, rw = t >> 7;
  const int xc = min(128, S), xs = xc >> 2;       // chunk, quarter
  const int split = xs >= dx_split<T>() ? dx_split<T>() : 1;
  const int hs = xs / split;                      // x per group and stage
  const int per = (S / xc) * split;               // stages per row set
  const int sx = 4 * hs;                          // x staged
  const size_t dbytes = static_cast<size_t>(kDxRows) * sx * C * sizeof(T);
  constexpr size_t kStage = dx_stage_bytes<T>();
  float2* red = reinterpret_cast<float2*>(dsm8 + 2 * kStage);  // [rows][16][C]
  const int sets = rows / kDxRows;
  const int mine = blockIdx.x < sets ? (sets - 1 - blockIdx.x) / gridDim.x + 1 : 0;
  // stage q of this block: row set q / per, step q % per; every length is a
  // power of two
  const int lhs = 31 - __clz(hs);
  auto issue = [&](int q) {
    const int set = q / per, st = q - set * per;
    const int r0 = (blockIdx.x + set * gridDim.x) * kDxRows;
    const int x0 = (st / split) * xc + (st % split) * hs;
    uint8_t* dst = dsm8 + (q & 1) * kStage;
    // [row][g hs + i][C]: x = x0 + g xs + i
    constexpr int kPer16 = 16 / sizeof(T), kVec = C / kPer16;  // 16-byte copies per x
    constexpr int lkVec = kVec == 8 ? 3 : 4;
    const T* src = in + (static_cast<size_t>(r0) * S + x0) * C;
    const int nvec = (kDxRows * kVec) << (lhs + 2);
    for (int e = t; e < nvec; e += kDxThreads) {
      const int v = e & (kVec - 1), xx = (e >> lkVec) & (sx - 1), row = e >> (lkVec + lhs + 2);
      const int x = (xx >> lhs) * xs + (xx & (hs - 1));
      cp16(dst + static_cast<size_t>(e) * 16, src + (static_cast<size_t>(row) * S + x) * C + v * kPer16);
    }
    for (int e = t; e < sx * 8; e += kDxThreads) {
      const int v = e & 7, xx = e >> 3;
      const int x = x0 + (xx >> lhs) * xs + (xx & (hs - 1));
      cp16(dst + dbytes + static_cast<size_t>(e) * 16, twt + static_cast<size_t>(x) * 16 + v * 2);
    }
    fr_cp_commit();
  };
  uint64_t acc[8][4];  // (re, im)
  const int total = mine * per;
  if (total > 0) issue(0);
  for (int q = 0, step = 0; q < total; ++q, step = step + 1 == per ? 0 : step + 1) {
    if (step == 0)
#pragma unroll
      for (int k = 0; k < 8; ++k)
#pragma unroll
        for (int c = 0; c < 4; ++c) acc[k][c] = 0;
    if (q + 1 < total) {
      issue(q + 1);
      fr_cp_wait<1>();
    } else {
      fr_cp_wait<0>();
    }
    __syncthreads();
    const uint8_t* st = dsm8 + (q & 1) * kStage;
    const T* a0 = reinterpret_cast<const T*>(st) + (static_cast<size_t>(rw) * sx + grp * hs) * C + cg * 4;
    const ulonglong2* w0 = reinterpret_cast<const ulonglong2*>(st + dbytes) + (grp * hs) * 8 + kg * 4;
#pragma unroll 4
    for (int i = 0; i < hs; ++i) {
      float a[4];
      load4(a0 + i * C, a);
      uint64_t a2[4];
#pragma unroll
      for (int c = 0; c < 4; ++c) a2[c] = pack2(a[c], a[c]);
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        const ulonglong2 w = w0[i * 8 + k];  // two modes' (cos, sin)
#pragma unroll
        for (int c = 0; c < 4; ++c) {
          fma2(acc[2 * k][c], a2[c], w.x);
          fma2(acc[2 * k + 1][c], a2[c], w.y);
        }
      }
    }
    if (step == per - 1) {
      // ((group 0 + 1) + 2) + 3 through shared memory
      const int r = (blockIdx.x + (q / per) * gridDim.x) * kDxRows + rw;
      for (int g = 0; g < 4; ++g) {
        if (grp == g) {
#pragma unroll
          for (int k = 0; k < 8; ++k) {
            const int kx = kg * 8 + k;
            float4* rp = reinterpret_cast<float4*>(red + (rw * 16 + kx) * C + cg * 4);
            const float2 c0 = unpack2(acc[k][0]), c1 = unpack2(acc[k][1]), c2 = unpack2(acc[k][2]),
                         c3 = unpack2(acc[k][3]);
            float4 lo = make_float4(c0.x, c0.y, c1.x, c1.y);
            float4 hi = make_float4(c2.x, c2.y, c3.x, c3.y);
            if (g > 0) {
              const float4 p = rp[0], s = rp[1];
              lo = make_float4(p.x + lo.x, p.y + lo.y, p.z + lo.z, p.w + lo.w);
              hi = make_float4(s.x + hi.x, s.y + hi.y, s.z + hi.z, s.w + hi.w);
            }
            if (g < 3) {
              rp[0] = lo;
              rp[1] = hi;
            } else if (kx < m) {
              float4* o = reinterpret_cast<float4*>(out + (static_cast<size_t>(r) * m + kx) * C + cg * 4);
              o[0] = lo;
              o[1] = hi;
            }
          }
        }
        if (g < 3) __syncthreads();
      }
    }
    __syncthreads();  // the stage's readers (and red's) before its next writers
  }
}

// ------------------------------------------------------------ DFT along y
// To modes: out[b][j][col] = sum_y in[b][y][col] w(j, y), col = (kx, c) over
// m C columns, J = 2m <= 32; tyt[y][32] holds the twiddles (zero past J).
// Order: y ascending, re = fma(x, wx, fma(-y, wy, re)), im = fma(x, wy,
// fma(y, wx, im)).
// 128 threads take 32 columns, a thread one column and eight modes; chunks of
// 32 y of input and twiddles by cp.async, two stages.  Bound by FP32 issue
// (32 multiply-adds for five shared loads); the kernel it replaces read every
// twiddle of every step from global memory, one per thread and mode:
// 16 x 512^2: 0.435 -> 0.062 ms.
constexpr int kDyY = 32;
__global__ void __launch_bounds__(128) fno_dft_y_fwd(const float2* __restrict__ in, int S, int m,
                                                      const float2* __restrict__ tyt, float2* __restrict__ out) {
  __shared__ __align__(16) float2 sv[2][kDyY][32];
  __shared__ __align__(16) float2 sw[2][kDyY][32];
  const int t = threadIdx.x, lane = t & 31, j0 = (t >> 5) * 8;
  const int J = 2 * m, mC = m * 64, b = blockIdx.y, col0 = blockIdx.x * 32;
  const int yc = min(kDyY, S), steps = S / yc;
  const float2* src = in + static_cast<size_t>(b) * S * mC + col0;
  auto issue = [&](int q) {
    for (int e = t; e < yc * 16; e += 128) {
      const int v = (e & 15) * 2, y = e >> 4;
      cp16(&sv[q & 1][y][v], src + static_cast<size_t>(q * yc + y) * mC + v);
      cp16(&sw[q & 1][y][v], tyt + static_cast<size_t>(q * yc + y) * 32 + v);
    }
    fr_cp_commit();
  };
  float2 acc[8];
#pragma unroll
  for (int q = 0; q < 8; ++q) acc[q] = make_float2(0.f, 0.f);
  issue(0);
  for (int q = 0; q < steps; ++q) {
    if (q + 1 < steps) {
      issue(q + 1);
      fr_cp_wait<1>();
    } else {
      fr_cp_wait<0>();
    }
    __syncthreads();
#pragma unroll 4
    for (int y = 0; y < yc; ++y) {
      const float2 v = sv[q & 1][y][lane];
      const float4* w4 = reinterpret_cast<const float4*>(&sw[q & 1][y][j0]);
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        const float4 w = w4[k];
        acc[2 * k].x = fmaf(v.x, w.x, fmaf(-v.y, w.y, acc[2 * k].x));
        acc[2 * k].y = fmaf(v.x, w.y, fmaf(v.y, w.x, acc[2 * k].y));
        acc[2 * k + 1].x = fmaf(v.x, w.z, fmaf(-v.y, w.w, acc[2 * k + 1].x));
        acc[2 * k + 1].y = fmaf(v.x, w.w, fmaf(v.y, w.z, acc[2 * k + 1].y));
      }
    }
    __syncthreads();
  }
#pragma unroll
  for (int k = 0; k < 8; ++k)
    if (j0 + k < J) out[(static_cast<size_t>(b) * J + j0 + k) * mC + col0 + lane] = acc[k];
}

// From modes: Z[b][y][col] = sum_j in[b][j][col] conj(w(j, y)), j ascending,
// each complex product formed and then added.  PACK writes the layer GEMM's
// BF16 operand instead: Zs[b S + y][c][2 kx], [2 kx + 1] = (w Re Z, -w Im Z),
// w = (kx ? 2 : 1) / S^2, 32 wide, zero for kk >= 2m.
// 128 threads take 128 columns (PACK: 16 kx x 8 c, so that a warp's stores
// are two 64-byte runs), each with its column's modes in registers, over a
// run of rows y whose twiddles sit in shared memory.  Bound by FP32 issue and
// the packed stores; the kernel it replaces re-read the modes and twiddles
// from global memory for every row, and the packing was a pass of its own:
// 16 x 512^2: 0.425 + 0.095 -> 0.102 ms.  `run` rows per block: 32, or 8 where
// that would leave SMs without a block.
constexpr int kDyRows = 32;
template <bool PACK>
__global__ void __launch_bounds__(128) fno_dft_y_inv(const float2* __restrict__ in, int S, int m,
                                                      const float2* __restrict__ tyt, int run,
                                                      float2* __restrict__ Z, __nv_bfloat16* __restrict__ Zs) {
  __shared__ __align__(16) float2 sw[kDyRows][32];
  const int t = threadIdx.x, b = blockIdx.z, y0 = blockIdx.y * run;
  const int J = 2 * m, mC = m * 64, ny = min(run, S - y0);
  const int kx = PACK ? (t & 15) : 0, c = PACK ? blockIdx.x * 8 + (t >> 4) : 0;
  const int col = PACK ? kx * 64 + c : blockIdx.x * 128 + t;
  const bool live = PACK ? kx < m : col < mC;
  for (int e = t; e < ny * 16; e += 128) {
    const int v = (e & 15) * 2, y = e >> 4;
    *reinterpret_cast<float4*>(&sw[y][v]) = *reinterpret_cast<const float4*>(tyt + static_cast<size_t>(y0 + y) * 32 + v);
  }
  float2 v[32];
#pragma unroll
  for (int q = 0; q < 32; ++q)
    v[q] = live && q < J ? in[(static_cast<size_t>(b) * J + q) * mC + col] : make_float2(0.f, 0.f);
  __syncthreads();
  const float inv = 1.f / (static_cast<float>(S) * S);
  const float wk = (kx == 0 ? 1.f : 2.f) * inv;
#pragma unroll 1
  for (int y = 0; y < ny; ++y) {
    float re = 0.f, im = 0.f;
#pragma unroll
    for (int q = 0; q < 32; q += 2) {
      if (q >= J) break;  // J is even: the padded modes add nothing
      const float4 w4 = *reinterpret_cast<const float4*>(&sw[y][q]);
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        float2 w = h ? make_float2(w4.z, w4.w) : make_float2(w4.x, w4.y);
        w.y = -w.y;
        re += v[q + h].x * w.x - v[q + h].y * w.y;
        im += v[q + h].x * w.y + v[q + h].y * w.x;
      }
    }
    const size_t r = static_cast<size_t>(b) * S + y0 + y;
    if (PACK) {
      __nv_bfloat162 o;
      o.x = __float2bfloat16_rn(wk * re);
      o.y = __float2bfloat16_rn(-wk * im);
      *reinterpret_cast<__nv_bfloat162*>(Zs + (r * 64 + c) * 32 + 2 * kx) = o;
    } else if (live) {
      Z[r * mC + col] = make_float2(re, im);
    }
  }
}

// ------------------------------------------------------------ lift
// v0[b][p][c] = Wl[c][0] a + Wl[c][1] x/S + Wl[c][2] y/S + bl[c], BF16.
// A thread keeps the weights of eight channels and writes 16 bytes per pixel;
// bound by the 128 bytes per pixel it writes (one 2-byte store and 64-bit
// index divisions per element before: 16 x 512^2: 1.36 -> 0.17 ms).
__global__ void __launch_bounds__(256) fno_lift(const float* __restrict__ a, int S, const float* __restrict__ Wl,
                                                 const float* __restrict__ bl, __nv_bfloat16* __restrict__ v,
                                                 int pixels) {
  const int c0 = (threadIdx.x & 7) * 8;
  float w0[8], w1[8], w2[8], b[8];
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    w0[i] = Wl[(c0 + i) * 3];
    w1[i] = Wl[(c0 + i) * 3 + 1];
    w2[i] = Wl[(c0 + i) * 3 + 2];
    b[i] = bl[c0 + i];
  }
  const unsigned SS = static_cast<unsigned>(S) * S;
  const int lgS = 31 - __clz(S);
  const float inv_s = 1.f / S;  // S is a power of two: the product is the quotient
  for (int bp = (blockIdx.x * 256 + threadIdx.x) >> 3; bp < pixels; bp += (gridDim.x * 256) >> 3) {
    const unsigned p = static_cast<unsigned>(bp) & (SS - 1);
    const float gx = static_cast<float>(p & (S - 1)) * inv_s, gy = static_cast<float>(p >> lgS) * inv_s;
    const float av = a[bp];
    __align__(16) __nv_bfloat16 o[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) o[i] = __float2bfloat16_rn(w0[i] * av + w1[i] * gx + w2[i] * gy + b[i]);
    *reinterpret_cast<uint4*>(v + static_cast<size_t>(bp) * 64 + c0) = *reinterpret_cast<const uint4*>(o);
  }
}

// Lift backward: dWl += sum dv0 (a, x/S, y/S), dbl += sum dv0, and the input
// gradient da[p] = sum_c Wl[c][0] dv0[p][c] (c ascending, one fused
// multiply-add per term).  Tiles of 64 pixels through shared memory: loaded
// with 16-byte accesses, summed over pixels by (channel, quarter of the tile)
// and over channels by pixel.  Bound by dv0's 256 bytes per pixel (a strided
// load per channel before: 8 x 512^2: 0.98 -> 0.11 ms).  Two blocks per SM:
// their atomics on the 256 sums take turns.
__global__ void __launch_bounds__(256) fno_lift_bwd(const float* __restrict__ a, const float* __restrict__ dv0, int S,
                                                     const float* __restrict__ Wl, int pixels,
                                                     float* __restrict__ dWl, float* __restrict__ dbl,
                                                     float* __restrict__ da) {
  constexpr int C = 64, LD = 65, PT = 64;
  __shared__ float sd[PT * LD];
  __shared__ float sa[PT], sw[C];
  __shared__ float red[4][C][4];
  const int t = threadIdx.x, c = t & 63, grp = t >> 6;
  if (t < C) sw[t] = Wl[t * 3];
  float s0 = 0.f, s1 = 0.f, s2 = 0.f, s3 = 0.f;
  const unsigned SS = static_cast<unsigned>(S) * S;
  const int lgS = 31 - __clz(S);
  const float inv_s = 1.f / S;
  const int tiles = pixels / PT;  // S >= 8: a multiple of 64 pixels
  float4 next[4];
  auto fetch = [&](int tile) {
#pragma unroll
    for (int i = 0; i < 4; ++i)
      next[i] = reinterpret_cast<const float4*>(dv0 + static_cast<size_t>(tile) * PT * C)[t + 256 * i];
  };
  if (blockIdx.x < tiles) fetch(blockIdx.x);
  for (int tile = blockIdx.x; tile < tiles; tile += gridDim.x) {
    __syncthreads();
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int e = (t + 256 * i) * 4, px = e >> 6, k = e & 63;
      sd[px * LD + k] = next[i].x;
      sd[px * LD + k + 1] = next[i].y;
      sd[px * LD + k + 2] = next[i].z;
      sd[px * LD + k + 3] = next[i].w;
    }
    if (t < PT) sa[t] = a[tile * PT + t];
    if (tile + static_cast<int>(gridDim.x) < tiles) fetch(tile + gridDim.x);
    __syncthreads();
#pragma unroll 4
    for (int i = 0; i < PT / 4; ++i) {
      const int px = grp * (PT / 4) + i;
      const unsigned p = static_cast<unsigned>(tile * PT + px) & (SS - 1);
      const float gx = static_cast<float>(p & (S - 1)) * inv_s, gy = static_cast<float>(p >> lgS) * inv_s;
      const float d = sd[px * LD + c];
      s0 += d * sa[px];
      s1 += d * gx;
      s2 += d * gy;
      s3 += d;
    }
    if (da && t < PT) {
      float acc = 0.f;
      for (int k = 0; k < C; ++k) acc += sw[k] * sd[t * LD + k];
      da[tile * PT + t] = acc;
    }
  }
  red[grp][c][0] = s0;
  red[grp][c][1] = s1;
  red[grp][c][2] = s2;
  red[grp][c][3] = s3;
  __syncthreads();
  if (t < C) {
    float q[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) q[i] = ((red[0][t][i] + red[1][t][i]) + red[2][t][i]) + red[3][t][i];
    atomicAdd(dWl + t * 3, q[0]);
    atomicAdd(dWl + t * 3 + 1, q[1]);
    atomicAdd(dWl + t * 3 + 2, q[2]);
    atomicAdd(dbl + t, q[3]);
  }
}

}  // namespace huv_dev

namespace huv_launch {

using namespace huv_dev;

namespace {
constexpr size_t kRedBytes = static_cast<size_t>(kDxRows) * 16 * 64 * sizeof(float2);
template <typename T>
cudaError_t dft_x(const T* in, int S, int m, const float2* twt, float2* out, int rows, cudaStream_t st) {
  static std::atomic<uint64_t> attr{0};
  constexpr size_t smem = 2 * dx_stage_bytes<T>() + kRedBytes;
  static_assert(smem <= 232448 / 2 - 1024, "fno_dft_x: shared memory");
  huv::once_per_device(attr, [] {
    huv::check_cuda(cudaFuncSetAttribute(fno_dft_x<T>, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(smem)),
                    "cudaFuncSetAttribute(fno_dft_x)");
  });
  int sms = 0, dev = 0;
  cudaError_t e;
  if ((e = cudaGetDevice(&dev)) != cudaSuccess) return e;
  if ((e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev)) != cudaSuccess) return e;
  fno_dft_x<T><<<std::min(rows / kDxRows, 2 * sms), kDxThreads, smem, st>>>(in, S, m, twt, out, rows);
  return cudaGetLastError();
}
}  // namespace

cudaError_t fno_dft_x_bf16(const __nv_bfloat16* in, int S, int m, const float2* twt, float2* out, int rows,
                           cudaStream_t st) {
  return dft_x(in, S, m, twt, out, rows, st);
}
cudaError_t fno_dft_x_f32(const float* in, int S, int m, const float2* twt, float2* out, int rows, cudaStream_t st) {
  return dft_x(in, S, m, twt, out, rows, st);
}
cudaError_t fno_dft_y(const float2* in, int B, int S, int m, const float2* tyt, float2* out, cudaStream_t st) {
  fno_dft_y_fwd<<<dim3(2 * m, B), 128, 0, st>>>(in, S, m, tyt, out);
  return cudaGetLastError();
}
// Z (float2, [b][y][kx][c]) or, with Zs, the packed BF16 operand of the tensor-core layer.
cudaError_t fno_idft_y(const float2* in, int B, int S, int m, const float2* tyt, float2* Z, __nv_bfloat16* Zs,
                       cudaStream_t st) {
  const int run = static_cast<long long>(8) * ((S + kDyRows - 1) / kDyRows) * B >= 148 ? kDyRows : 8;
  const unsigned ry = (S + run - 1) / run;
  if (Zs)
    fno_dft_y_inv<true><<<dim3(8, ry, B), 128, 0, st>>>(in, S, m, tyt, run, nullptr, Zs);
  else
    fno_dft_y_inv<false><<<dim3((m * 64 + 127) / 128, ry, B), 128, 0, st>>>(in, S, m, tyt, run, Z, nullptr);
  return cudaGetLastError();
}
cudaError_t fno_lift_fwd(const float* a, int B, int S, const float* Wl, const float* bl, __nv_bfloat16* v,
                         cudaStream_t st) {
  const size_t pix = static_cast<size_t>(B) * S * S;
  fno_lift<<<static_cast<unsigned>(std::min<size_t>((pix + 31) / 32, 148 * 16)), 256, 0, st>>>(a, S, Wl, bl, v,
                                                                                              static_cast<int>(pix));
  return cudaGetLastError();
}
cudaError_t fno_lift_back(const float* a, const float* dv0, int B, int S, const float* Wl, float* dWl, float* dbl,
                          float* da, cudaStream_t st) {
  const size_t pix = static_cast<size_t>(B) * S * S;
  fno_lift_bwd<<<static_cast<unsigned>(std::min<size_t>(pix / 64, 148 * 2)), 256, 0, st>>>(
      a, dv0, S, Wl, static_cast<int>(pix), dWl, dbl, da);
  return cudaGetLastError();
}

}  // namespace huv_launch
