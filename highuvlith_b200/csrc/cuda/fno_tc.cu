// tcgen05 channel GEMMs of the FNO (grids of at least 128).
//
// The pointwise layer and the projection head are contractions over the 64
// channels of every pixel: [pixels x 64] x [64 x N].  Pixels are tiled by
// 128 (one tile never crosses an image row when the grid is >= 128); the
// channels-last BF16 activations of a tile are one 128 x 128-byte TMA box
// (128B swizzle, K-major), the weights are resident in shared memory.
//
// fno_tc_layer: D[p][o] = sum_i v[p][i] W[o][i]
//                       + sum_kk Tw[x(p)][kk] Zs[row(p)][o][kk]
// where the second term is the layer's inverse x-DFT of the retained modes
// (Tw[x][2kx] = cos, Tw[x][2kx+1] = sin of 2 pi kx x / S; Zs = (w_kx / S^2)
// (Re Z, -Im Z) per image row; 32 wide), folded in as a second K block.
// Epilogue: z = D + b, z stored (BF16) when a backward pass will follow,
// v_next = GELU(z).
// fno_tc_proj: D[p][j] = sum_i v[p][i] Q1[j][i], j < 128; epilogue
// out[p] = sum_j Q2[j] GELU(D[p][j] + b1[j]) + b2, one pixel per thread.
//
// Warp roles: 0 TMA producer (no multicast), 1 MMA issuer (one thread), then
// the epilogue warps.  Two shared-memory stages, tensor memory
// double-buffered, two CTAs per SM.  Every mbarrier wait is bounded
// (2 s); a timeout sets *err and unwinds.  Operands BF16, accumulation FP32.
#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include "../engine.hpp"
#include "fno_gelu.cuh"
#include "tc_ptx.cuh"

namespace huv_dev {

constexpr int kFnoStages = 2;  // two stages keep two CTAs (8 epilogue warps) per SM
constexpr uint64_t kFnoWaitNs = 2000000000ull;
constexpr uint32_t kTile = 128 * 128;  // 128 rows x 64 bf16

struct FnoTcParams {
  int tiles;          // 128-pixel tiles
  int S;              // grid side
  int kk_steps;       // layer: 16-wide K steps of the spectral block (ceil(2m / 16))
  const float* bias;  // layer: b[64]; projection: b1[128]
  const float* q2;    // projection: Q2[128]
  const float* b2;    // projection: b2[1]
  int act;            // layer: GELU on v_next
  int save_z;         // layer: z is stored
  float* out;         // projection
  int* err;
};

// Eight epilogue warps, two per tensor-memory lane quadrant (each 32 of the
// 64 channels of its pixels); a warp stages its 32 pixels x 32 channels in
// shared memory (64B swizzle) and stores them with TMA.  Bound by the
// epilogue's instructions, GELU above all, beside 256 bytes per pixel (384
// with z).  16 x 512^2: 0.68 -> 0.31 ms (3.4 TB/s); 8 x 512^2 with z: 0.345 ->
// 0.177 ms, with two erff per pair, four epilogue warps, 16-byte stores a
// pixel apart and z always written before.
constexpr int kFnoEpiWarps = 8;
constexpr uint32_t kFnoLayerStage = kTile + 128 * 64 + 64 * 64;  // v, twiddles, Zs
constexpr uint32_t kFnoOutTile = 32 * 64;                        // 32 pixels x 32 bf16
constexpr size_t kFnoLayerSmem =
    1024 + 64 * 128 + kFnoStages * kFnoLayerStage + kFnoEpiWarps * 2 * kFnoOutTile + 64 * 4 + 256;

__global__ void __launch_bounds__(32 * (2 + kFnoEpiWarps), 2)
    fno_tc_layer(const __grid_constant__ CUtensorMap tmV, const __grid_constant__ CUtensorMap tmW,
                 const __grid_constant__ CUtensorMap tmTw, const __grid_constant__ CUtensorMap tmZ,
                 const __grid_constant__ CUtensorMap tmVn, const __grid_constant__ CUtensorMap tmZo, FnoTcParams p) {
  constexpr int N = 64;
  constexpr uint32_t kWBytes = N * 128;
  extern __shared__ uint8_t smem_raw[];
  const uint32_t raw = smem_u32(smem_raw);
  uint8_t* base = smem_raw + (((raw + 1023u) & ~1023u) - raw);
  uint8_t* sW = base;
  uint8_t* sS = base + kWBytes;
  uint8_t* sO = sS + kFnoStages * kFnoLayerStage;  // [warp][v, z]
  float* sb = reinterpret_cast<float*>(sO + kFnoEpiWarps * 2 * kFnoOutTile);
  uint64_t* bars = reinterpret_cast<uint64_t*>(sb + 64);
  uint64_t* full = bars;
  uint64_t* empty = bars + kFnoStages;
  uint64_t* w_full = bars + 2 * kFnoStages;
  uint64_t* tfull = bars + 2 * kFnoStages + 1;
  uint64_t* tempty = bars + 2 * kFnoStages + 3;
  uint64_t* done = bars + 2 * kFnoStages + 5;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 2 * kFnoStages + 6);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  constexpr uint32_t kTmemCols = 128;

  if (threadIdx.x == 0) {
    for (int s = 0; s < kFnoStages; ++s) {
      mbar_init(&full[s], 1);
      mbar_init(&empty[s], 1);
    }
    mbar_init(w_full, 1);
    mbar_init(&tfull[0], 1);
    mbar_init(&tfull[1], 1);
    mbar_init(&tempty[0], kFnoEpiWarps);
    mbar_init(&tempty[1], kFnoEpiWarps);
    mbar_init(done, 1);
    *abort_flag = 0;
    fence_barrier_init();
  }
  if (threadIdx.x < 64) sb[threadIdx.x] = p.bias[threadIdx.x];
  if (warp == 0) {
    tmem_alloc(tmem_slot, kTmemCols);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  auto fail = [&](int code) {
    *abort_flag = 1;
    if (p.err) atomicExch(p.err, code);
  };
  const int SS = p.S * p.S;

  if (warp == 0) {
    if (lane == 0) {
      prefetch_tmap(&tmV);
      prefetch_tmap(&tmW);
      mbar_arrive_expect_tx(w_full, kWBytes);
      tma_load_2d(sW, &tmW, 0, 0, w_full);
      int it = 0;
      for (int t = blockIdx.x; t < p.tiles && !*abort_flag; t += gridDim.x, ++it) {
        const int s = it % kFnoStages;
        if (!mbar_wait_or_abort(&empty[s], ((it / kFnoStages) & 1) ^ 1, kFnoWaitNs, abort_flag)) {
          fail(11);
          break;
        }
        uint8_t* st = sS + s * kFnoLayerStage;
        const int p0 = t * 128;
        mbar_arrive_expect_tx(&full[s], kFnoLayerStage);
        tma_load_2d(st, &tmV, 0, p0, &full[s]);
        const int b = p0 / SS, rem = p0 - b * SS, y = rem / p.S, x0 = rem - y * p.S;
        tma_load_2d(st + kTile, &tmTw, 0, x0, &full[s]);
        tma_load_2d(st + kTile + 128 * 64, &tmZ, 0, (b * p.S + y) * 64, &full[s]);
      }
      // every load issued lands before the CTA may exit
      mbar_wait(w_full, 0, kFnoWaitNs);
      for (int q = (it > kFnoStages ? it - kFnoStages : 0); q < it; ++q)
        mbar_wait(&full[q % kFnoStages], (q / kFnoStages) & 1, kFnoWaitNs);
    }
  } else if (warp == 1) {
    if (lane == 0) {
      const uint32_t idesc = idesc_bf16(128, N);
      bool ok = mbar_wait(w_full, 0, kFnoWaitNs);
      if (!ok) fail(12);
      tc_fence_after();
      int it = 0;
      for (int t = blockIdx.x; t < p.tiles && ok && !*abort_flag; t += gridDim.x, ++it) {
        const int s = it % kFnoStages, buf = it & 1;
        if (!mbar_wait_or_abort(&tempty[buf], ((it >> 1) & 1) ^ 1, kFnoWaitNs, abort_flag)) {
          fail(13);
          break;
        }
        if (!mbar_wait(&full[s], (it / kFnoStages) & 1, kFnoWaitNs)) {
          fail(14);
          break;
        }
        tc_fence_after();
        const uint32_t d = tmem_base + buf * N;
        uint8_t* st = sS + s * kFnoLayerStage;
        const uint64_t av = smem_desc_sw128(smem_u32(st));
        const uint64_t bw = smem_desc_sw128(smem_u32(sW));
#pragma unroll
        for (int ks = 0; ks < 4; ++ks) tc_mma_bf16(d, av + 2 * ks, bw + 2 * ks, idesc, ks > 0 ? 1u : 0u);
        const uint64_t at = smem_desc_sw64(smem_u32(st + kTile));
        const uint64_t bz = smem_desc_sw64(smem_u32(st + kTile + 128 * 64));
        for (int ks = 0; ks < p.kk_steps; ++ks) tc_mma_bf16(d, at + 2 * ks, bz + 2 * ks, idesc, 1u);
        tc_commit(&empty[s]);
        tc_commit(&tfull[buf]);
      }
      tc_commit(done);
      mbar_wait(done, 0, kFnoWaitNs);
    }
  } else {
    const int quad = warp & 3, c0 = ((warp - 2) >> 2) * 32;
    uint8_t* ov = sO + (warp - 2) * 2 * kFnoOutTile;
    const uint32_t sw = static_cast<uint32_t>(lane >> 1) & 3u;  // 64B swizzle of row `lane`
    int it = 0;
    for (int t = blockIdx.x; t < p.tiles; t += gridDim.x, ++it) {
      const int buf = it & 1;
      const bool got =
          __all_sync(0xffffffffu, mbar_wait_or_abort(&tfull[buf], (it >> 1) & 1, kFnoWaitNs, abort_flag));
      if (!got) {
        if (lane == 0) fail(15);
        break;
      }
      tc_fence_after();
      float v[32];
      tmem_ld32(tmem_base + (static_cast<uint32_t>(quad * 32) << 16) + buf * N + c0, v);
      tc_fence_before();
      __syncwarp();
      if (lane == 0) {
        mbar_arrive(&tempty[buf]);
        // v_next alternates between the two buffers, or leaves the second to z
        if (p.save_z)
          bulk_wait_read<0>();
        else
          bulk_wait_read<1>();
      }
      __syncwarp();
      uint8_t* dv = ov + (p.save_z || !(it & 1) ? 0 : kFnoOutTile) + lane * 64;
      uint8_t* dz = ov + kFnoOutTile + lane * 64;
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        const float4 ba = *reinterpret_cast<const float4*>(sb + c0 + 8 * q);
        const float4 bb = *reinterpret_cast<const float4*>(sb + c0 + 8 * q + 4);
        const float z[8] = {v[8 * q] + ba.x,     v[8 * q + 1] + ba.y, v[8 * q + 2] + ba.z, v[8 * q + 3] + ba.w,
                            v[8 * q + 4] + bb.x, v[8 * q + 5] + bb.y, v[8 * q + 6] + bb.z, v[8 * q + 7] + bb.w};
        uint32_t zw[4], vw[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const __nv_bfloat162 zb = __floats2bfloat162_rn(z[2 * i], z[2 * i + 1]);
          const __nv_bfloat162 vb = p.act ? gelu_bf16x2(z[2 * i], z[2 * i + 1]) : zb;
          zw[i] = *reinterpret_cast<const uint32_t*>(&zb);
          vw[i] = *reinterpret_cast<const uint32_t*>(&vb);
        }
        const uint32_t o = (static_cast<uint32_t>(q) ^ sw) << 4;
        *reinterpret_cast<uint4*>(dv + o) = make_uint4(vw[0], vw[1], vw[2], vw[3]);
        if (p.save_z) *reinterpret_cast<uint4*>(dz + o) = make_uint4(zw[0], zw[1], zw[2], zw[3]);
      }
      fence_proxy_async_smem();
      __syncwarp();
      if (lane == 0) {
        tma_store_2d(&tmVn, dv, c0, t * 128 + quad * 32);
        if (p.save_z) tma_store_2d(&tmZo, dz, c0, t * 128 + quad * 32);
        bulk_commit();
      }
    }
    // every TMA store must have finished before the CTA's shared memory goes
    if (lane == 0 && it > 0) bulk_wait<0>();
    __syncwarp();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  if (warp == 0) tmem_dealloc(tmem_base, kTmemCols);
}

// Projection: eight epilogue warps, warps 2..5 the even tiles of the CTA and
// 6..9 the odd ones (a pixel's sum over the 128 hidden units runs in one
// thread, in order).  Bound by erff: 128 GELUs per pixel beside 132 bytes;
// 16 x 512^2: 0.84 -> 0.57 ms with twice the epilogue warps and the biases
// read four at a time.
constexpr size_t kFnoProjSmem = 1024 + 128 * 128 + kFnoStages * kTile + 2 * 128 * 4 + 256;

__global__ void __launch_bounds__(32 * (2 + kFnoEpiWarps), 2)
    fno_tc_proj(const __grid_constant__ CUtensorMap tmV, const __grid_constant__ CUtensorMap tmW, FnoTcParams p) {
  constexpr int N = 128;
  constexpr uint32_t kWBytes = N * 128;
  extern __shared__ uint8_t smem_raw[];
  const uint32_t raw = smem_u32(smem_raw);
  uint8_t* base = smem_raw + (((raw + 1023u) & ~1023u) - raw);
  uint8_t* sW = base;
  uint8_t* sS = base + kWBytes;
  float* sb = reinterpret_cast<float*>(sS + kFnoStages * kTile);  // b1[128], Q2[128]
  uint64_t* bars = reinterpret_cast<uint64_t*>(sb + 2 * N);
  uint64_t* full = bars;
  uint64_t* empty = bars + kFnoStages;
  uint64_t* w_full = bars + 2 * kFnoStages;
  uint64_t* tfull = bars + 2 * kFnoStages + 1;
  uint64_t* tempty = bars + 2 * kFnoStages + 3;
  uint64_t* done = bars + 2 * kFnoStages + 5;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 2 * kFnoStages + 6);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  constexpr uint32_t kTmemCols = 256;

  if (threadIdx.x == 0) {
    for (int s = 0; s < kFnoStages; ++s) {
      mbar_init(&full[s], 1);
      mbar_init(&empty[s], 1);
    }
    mbar_init(w_full, 1);
    mbar_init(&tfull[0], 1);
    mbar_init(&tfull[1], 1);
    mbar_init(&tempty[0], 4);
    mbar_init(&tempty[1], 4);
    mbar_init(done, 1);
    *abort_flag = 0;
    fence_barrier_init();
  }
  if (threadIdx.x < 128)
    sb[threadIdx.x] = p.bias[threadIdx.x];
  else if (threadIdx.x < 256)
    sb[threadIdx.x] = p.q2[threadIdx.x - 128];
  if (warp == 0) {
    tmem_alloc(tmem_slot, kTmemCols);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  auto fail = [&](int code) {
    *abort_flag = 1;
    if (p.err) atomicExch(p.err, code);
  };

  if (warp == 0) {
    if (lane == 0) {
      prefetch_tmap(&tmV);
      prefetch_tmap(&tmW);
      mbar_arrive_expect_tx(w_full, kWBytes);
      tma_load_2d(sW, &tmW, 0, 0, w_full);
      int it = 0;
      for (int t = blockIdx.x; t < p.tiles && !*abort_flag; t += gridDim.x, ++it) {
        const int s = it % kFnoStages;
        if (!mbar_wait_or_abort(&empty[s], ((it / kFnoStages) & 1) ^ 1, kFnoWaitNs, abort_flag)) {
          fail(11);
          break;
        }
        mbar_arrive_expect_tx(&full[s], kTile);
        tma_load_2d(sS + s * kTile, &tmV, 0, t * 128, &full[s]);
      }
      // every load issued lands before the CTA may exit
      mbar_wait(w_full, 0, kFnoWaitNs);
      for (int q = (it > kFnoStages ? it - kFnoStages : 0); q < it; ++q)
        mbar_wait(&full[q % kFnoStages], (q / kFnoStages) & 1, kFnoWaitNs);
    }
  } else if (warp == 1) {
    if (lane == 0) {
      const uint32_t idesc = idesc_bf16(128, N);
      bool ok = mbar_wait(w_full, 0, kFnoWaitNs);
      if (!ok) fail(12);
      tc_fence_after();
      int it = 0;
      for (int t = blockIdx.x; t < p.tiles && ok && !*abort_flag; t += gridDim.x, ++it) {
        const int s = it % kFnoStages, buf = it & 1;
        if (!mbar_wait_or_abort(&tempty[buf], ((it >> 1) & 1) ^ 1, kFnoWaitNs, abort_flag)) {
          fail(13);
          break;
        }
        if (!mbar_wait(&full[s], (it / kFnoStages) & 1, kFnoWaitNs)) {
          fail(14);
          break;
        }
        tc_fence_after();
        const uint64_t av = smem_desc_sw128(smem_u32(sS + s * kTile));
        const uint64_t bw = smem_desc_sw128(smem_u32(sW));
#pragma unroll
        for (int ks = 0; ks < 4; ++ks)
          tc_mma_bf16(tmem_base + buf * N, av + 2 * ks, bw + 2 * ks, idesc, ks > 0 ? 1u : 0u);
        tc_commit(&empty[s]);
        tc_commit(&tfull[buf]);
      }
      tc_commit(done);
      mbar_wait(done, 0, kFnoWaitNs);
    }
  } else {
    const int quad = warp & 3, par = (warp - 2) >> 2;
    const float b2 = __ldg(p.b2);
    int it = 0;
    for (int t = blockIdx.x; t < p.tiles; t += gridDim.x, ++it) {
      if ((it & 1) != par) continue;
      const int buf = it & 1;
      const bool got =
          __all_sync(0xffffffffu, mbar_wait_or_abort(&tfull[buf], (it >> 1) & 1, kFnoWaitNs, abort_flag));
      if (!got) {
        if (lane == 0) fail(15);
        break;
      }
      tc_fence_after();
      const uint32_t taddr = tmem_base + (static_cast<uint32_t>(quad * 32) << 16) + buf * N;
      float acc = b2;
#pragma unroll 1
      for (int c0 = 0; c0 < N; c0 += 32) {
        float v[32];
        tmem_ld32(taddr + c0, v);
#pragma unroll
        for (int i = 0; i < 32; i += 4) {
          const float4 bj = *reinterpret_cast<const float4*>(sb + c0 + i);
          const float4 qj = *reinterpret_cast<const float4*>(sb + N + c0 + i);
          acc += qj.x * gelu_erf(v[i] + bj.x);
          acc += qj.y * gelu_erf(v[i + 1] + bj.y);
          acc += qj.z * gelu_erf(v[i + 2] + bj.z);
          acc += qj.w * gelu_erf(v[i + 3] + bj.w);
        }
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&tempty[buf]);
      p.out[static_cast<size_t>(t) * 128 + quad * 32 + lane] = acc;
    }
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  if (warp == 0) tmem_dealloc(tmem_base, kTmemCols);
}

// ------------------------------------------------------------------ backward
// Backward of the pointwise layer on tcgen05, per 128-pixel tile:
//   dz = dvnext * GELU'(z)  (or dvnext for the last layer), stored (f32);
//   dv = dz W               (M 128 pixels, N 64 inputs, K 64 outputs), stored (f32);
//   dW += dz^T v, db += sum dz over the CTA's tiles.
// The elementwise part runs on CUDA cores (warps 6..13; eight lanes take the
// eight 8-channel octets of a pixel, so that a warp reads and writes whole
// 256-byte rows) and writes dz as BF16 into shared memory in the 128B-swizzled
// layout of a pixel row of 64 channels, where both GEMMs read it: K-major
// [px][o] for dv, and MN-major (the same bytes, pixels as K) for dW, whose
// other operand is the v tile as TMA loads it, MN-major too.  dW is the top
// half of the 128 x 64 product (dz^T; v^T) v, accumulated in tensor memory
// over every tile of the CTA and added to global memory once.  Warp 0 issues
// the MMAs (one thread), warp 1 loads v, warps 2..5 drain dv from tensor
// memory and store it with TMA.  Operand stages and dv accumulators are
// double-buffered; two CTAs per SM, persistent.  Every mbarrier wait is
// bounded; a timeout sets *err and unwinds.
//
// What bounds it: 1 KB per pixel, and GELU' (erff and expf).  With one pixel
// per lane (32 rows of 16 bytes per access) and operands transposed by 2-byte
// stores it was bound by L1 (87 %), 0.66 ms at 8 x 512^2; now 0.36 ms.
constexpr int kBwdXWarps = 8;                       // elementwise warps
constexpr int kBwdThreads = 32 * (6 + kBwdXWarps);  // MMA + TMA + 4 epilogue + elementwise
constexpr uint32_t kBwdStage = 2 * 16384;           // dz [128 px][64 o], v [128 px][64 i]
constexpr uint32_t kBwdOut = 32 * 32 * 4;           // dv staging tile: 32 px x 32 channels
constexpr size_t kBwdSmem = 1024 + 8192 + 2 * static_cast<size_t>(kBwdStage) + 4 * 2 * kBwdOut + 256;

__device__ __forceinline__ float tc_gelu_grad(float x) {
  const float cdf = 0.5f * (1.f + erff(x * 0.70710678118654752f));
  const float pdf = 0.39894228040143268f * expf(-0.5f * x * x);
  return cdf + x * pdf;
}

// byte offset of element (row, k) in a K-major 128B-swizzled tile of 128-byte rows
__device__ __forceinline__ uint32_t sw128_off(int row, int k) {
  return static_cast<uint32_t>(row) * 128u + ((static_cast<uint32_t>(k >> 3) ^ static_cast<uint32_t>(row & 7)) << 4) +
         static_cast<uint32_t>(k & 7) * 2u;
}

struct FnoBwdParams {
  int tiles;
  int act;
  const float* dvnext;      // [pix][64]
  const __nv_bfloat16* z;   // [pix][64]
  const float* W;           // [64 o][64 i]
  float* dz;                // [pix][64]
  float* dW;                // [64][64], accumulated
  float* db;                // [64], accumulated
  int* err;
};

__global__ void __launch_bounds__(kBwdThreads, 2)
    fno_tc_layer_bwd(const __grid_constant__ CUtensorMap tmV, const __grid_constant__ CUtensorMap tmDv, FnoBwdParams p) {
  extern __shared__ uint8_t smem_raw[];
  const uint32_t raw = smem_u32(smem_raw);
  uint8_t* base = smem_raw + (((raw + 1023u) & ~1023u) - raw);
  uint8_t* sWT = base;               // [64 i][64 o]
  uint8_t* sS = base + 8192;         // [stage] { dz, v }
  uint8_t* sO = sS + 2 * kBwdStage;  // [epilogue warp][2]
  uint64_t* bars = reinterpret_cast<uint64_t*>(sO + 4 * 2 * kBwdOut);
  uint64_t* full = bars;             // [2], one arrival per elementwise warp
  uint64_t* vfull = bars + 2;        // [2], TMA
  uint64_t* empty = bars + 4;        // [2], MMA commit
  uint64_t* tfull = bars + 6;        // [2]
  uint64_t* tempty = bars + 8;       // [2], one arrival per epilogue warp
  uint64_t* done = bars + 10;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 11);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  __shared__ float sdb[kBwdXWarps * 64];
  constexpr uint32_t kTmemCols = 256;  // dv accumulators at 0 / 64, dW at 128

  if (threadIdx.x == 0) {
    for (int s = 0; s < 2; ++s) {
      mbar_init(&full[s], kBwdXWarps);
      mbar_init(&vfull[s], 1);
      mbar_init(&empty[s], 1);
      mbar_init(&tfull[s], 1);
      mbar_init(&tempty[s], 4);
    }
    mbar_init(done, 1);
    *abort_flag = 0;
    fence_barrier_init();
  }
  if (warp == 0) {
    tmem_alloc(tmem_slot, kTmemCols);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  auto fail = [&](int code) {
    *abort_flag = 1;
    if (p.err) atomicExch(p.err, code);
  };

  if (warp == 0) {
    if (lane == 0) {
      const uint32_t idk = idesc_bf16(128, 64), idm = idk | kIdescAMn | kIdescBMn;
      const uint64_t bw = smem_desc_sw128(smem_u32(sWT));
      int it = 0;
      for (int t = blockIdx.x; t < p.tiles && !*abort_flag; t += gridDim.x, ++it) {
        const int s = it & 1;
        const uint32_t ph = (it >> 1) & 1;
        if (!mbar_wait_or_abort(&tempty[s], ph ^ 1, kFnoWaitNs, abort_flag)) {
          fail(31);
          break;
        }
        if (!mbar_wait_or_abort(&full[s], ph, kFnoWaitNs, abort_flag) ||
            !mbar_wait_or_abort(&vfull[s], ph, kFnoWaitNs, abort_flag)) {
          fail(32);
          break;
        }
        tc_fence_after();
        const uint32_t sA = smem_u32(sS + s * kBwdStage), sV = sA + 16384;
        const uint64_t aa = smem_desc_sw128(sA);
#pragma unroll
        for (int ks = 0; ks < 4; ++ks) tc_mma_bf16(tmem_base + s * 64, aa + 2 * ks, bw + 2 * ks, idk, ks > 0 ? 1u : 0u);
        tc_commit(&tfull[s]);
        // rows 0..63: dz^T, rows 64..127: v^T (the v tile follows dz's)
        const uint64_t ax = smem_desc_sw128_mn(sA, 16384), bx = smem_desc_sw128_mn(sV, 16384);
#pragma unroll
        for (int ks = 0; ks < 8; ++ks)
          tc_mma_bf16(tmem_base + 128, ax + kMnStep * ks, bx + kMnStep * ks, idm, (it > 0 || ks > 0) ? 1u : 0u);
        tc_commit(&empty[s]);
      }
      tc_commit(done);
      mbar_wait(done, 0, kFnoWaitNs);
    }
  } else if (warp == 1) {
    if (lane == 0) {
      prefetch_tmap(&tmV);
      prefetch_tmap(&tmDv);
      int it = 0;
      for (int t = blockIdx.x; t < p.tiles && !*abort_flag; t += gridDim.x, ++it) {
        const int s = it & 1;
        if (!mbar_wait_or_abort(&empty[s], ((it >> 1) & 1) ^ 1, kFnoWaitNs, abort_flag)) {
          fail(36);
          break;
        }
        mbar_arrive_expect_tx(&vfull[s], kTile);
        tma_load_2d(sS + s * kBwdStage + 16384, &tmV, 0, t * 128, &vfull[s]);
      }
      // every load issued lands before the CTA may exit
      for (int q = (it > 2 ? it - 2 : 0); q < it; ++q) mbar_wait(&vfull[q & 1], (q >> 1) & 1, kFnoWaitNs);
    }
  } else if (warp <= 5) {
    // dv epilogue: lane quadrant warp % 4, one pixel row per lane
    const int quad = warp & 3;
    uint8_t* st = sO + quad * 2 * kBwdOut;
    int it = 0;
    for (int t = blockIdx.x; t < p.tiles; t += gridDim.x, ++it) {
      const int s = it & 1;
      const bool got =
          __all_sync(0xffffffffu, mbar_wait_or_abort(&tfull[s], (it >> 1) & 1, kFnoWaitNs, abort_flag));
      if (!got) {
        if (lane == 0) fail(33);
        break;
      }
      tc_fence_after();
      const uint32_t taddr = tmem_base + (static_cast<uint32_t>(quad * 32) << 16) + s * 64;
#pragma unroll 1
      for (int h = 0; h < 2; ++h) {
        float a[32];
        tmem_ld32(taddr + 32 * h, a);
        if (h == 1) {
          tc_fence_before();
          __syncwarp();
          if (lane == 0) mbar_arrive(&tempty[s]);
        }
        if (lane == 0) bulk_wait_read<1>();  // this half's buffer was last stored one tile ago
        __syncwarp();
        uint8_t* o = st + h * kBwdOut;
#pragma unroll
        for (int q = 0; q < 8; ++q)
          *reinterpret_cast<float4*>(o + lane * 128 + ((q ^ (lane & 7)) << 4)) =
              make_float4(a[4 * q], a[4 * q + 1], a[4 * q + 2], a[4 * q + 3]);
        fence_proxy_async_smem();
        __syncwarp();
        if (lane == 0) {
          tma_store_2d(&tmDv, o, 32 * h, t * 128 + quad * 32);
          bulk_commit();
        }
      }
    }
    if (lane == 0 && it > 0) bulk_wait<0>();
    __syncwarp();
    // dW rows o = lanes 0..63 of the second accumulator, once every MMA is complete
    if (quad < 2) {
      const bool fin = __all_sync(0xffffffffu, mbar_wait(done, 0, kFnoWaitNs));
      if (__all_sync(0xffffffffu, fin && !*abort_flag)) {  // one finding per warp: tcgen05.ld is .sync.aligned
        tc_fence_after();
        const uint32_t taddr = tmem_base + (static_cast<uint32_t>(quad * 32) << 16) + 128;
        // through the staging tiles, so that a warp's atomics cover 128
        // consecutive bytes (a row per lane: 8 times the L2 operations, 0.1 ms
        // of every launch for 296 CTAs)
#pragma unroll 1
        for (int h = 0; h < 2; ++h) {
          float a[32];
          tmem_ld32(taddr + 32 * h, a);
          uint8_t* o = st + h * kBwdOut;
#pragma unroll
          for (int q = 0; q < 8; ++q)
            *reinterpret_cast<float4*>(o + lane * 128 + ((q ^ (lane & 7)) << 4)) =
                make_float4(a[4 * q], a[4 * q + 1], a[4 * q + 2], a[4 * q + 3]);
          __syncwarp();
          float* w = p.dW + quad * 32 * 64 + 32 * h + lane;
#pragma unroll 8
          for (int r = 0; r < 32; ++r)
            atomicAdd(w + r * 64, *reinterpret_cast<const float*>(o + r * 128 + (((lane >> 2) ^ (r & 7)) << 4) + (lane & 3) * 4));
        }
      } else if (!fin && lane == 0) {
        fail(34);
      }
    }
  } else {
    // elementwise warps: lane = (pixel of four, octet of channels)
    const int xw = warp - 6, o0 = 8 * (lane & 7);
    const int xt = threadIdx.x - 6 * 32;
    // W^T into sWT once: element (o, i) of W is row i, column o of the B operand
    for (int e = xt; e < 64 * 64; e += 32 * kBwdXWarps) {
      const int o = e >> 6, i = e & 63;
      *reinterpret_cast<__nv_bfloat16*>(sWT + sw128_off(i, o)) = __float2bfloat16_rn(p.W[e]);
    }
    float dbp[8];
#pragma unroll
    for (int e = 0; e < 8; ++e) dbp[e] = 0.f;
    int it = 0;
    for (int t = blockIdx.x; t < p.tiles; t += gridDim.x, ++it) {
      const int s = it & 1;
      uint8_t* sA = sS + s * kBwdStage;
      bool ok = true;
#pragma unroll 1
      for (int h = 0; h < 2; ++h) {
        float4 g[2][2];
        uint4 zz[2];
#pragma unroll
        for (int c = 0; c < 2; ++c) {
          const int px = 16 * xw + 8 * h + 4 * c + (lane >> 3);
          const size_t off = (static_cast<size_t>(t) * 128 + px) * 64 + o0;
          g[c][0] = *reinterpret_cast<const float4*>(p.dvnext + off);
          g[c][1] = *reinterpret_cast<const float4*>(p.dvnext + off + 4);
          zz[c] = p.act ? *reinterpret_cast<const uint4*>(p.z + off) : make_uint4(0, 0, 0, 0);
        }
        if (h == 0)  // stage s was last read by the MMAs of tile it - 2
          ok = __all_sync(0xffffffffu, mbar_wait_or_abort(&empty[s], ((it >> 1) & 1) ^ 1, kFnoWaitNs, abort_flag));
        if (!ok) break;
#pragma unroll
        for (int c = 0; c < 2; ++c) {
          const int px = 16 * xw + 8 * h + 4 * c + (lane >> 3);
          const size_t off = (static_cast<size_t>(t) * 128 + px) * 64 + o0;
          const float gv[8] = {g[c][0].x, g[c][0].y, g[c][0].z, g[c][0].w, g[c][1].x, g[c][1].y, g[c][1].z, g[c][1].w};
          const __nv_bfloat16* zb = reinterpret_cast<const __nv_bfloat16*>(&zz[c]);
          float d[8];
#pragma unroll
          for (int e = 0; e < 8; ++e) {
            d[e] = p.act ? gv[e] * tc_gelu_grad(__bfloat162float(zb[e])) : gv[e];
            dbp[e] += d[e];
          }
          reinterpret_cast<float4*>(p.dz + off)[0] = make_float4(d[0], d[1], d[2], d[3]);
          reinterpret_cast<float4*>(p.dz + off)[1] = make_float4(d[4], d[5], d[6], d[7]);
          __align__(16) __nv_bfloat16 db16[8];
#pragma unroll
          for (int e = 0; e < 8; ++e) db16[e] = __float2bfloat16_rn(d[e]);
          *reinterpret_cast<uint4*>(sA + sw128_off(px, o0)) = *reinterpret_cast<const uint4*>(db16);
        }
      }
      if (!ok) {
        if (lane == 0) fail(35);
        break;
      }
      fence_proxy_async_smem();
      __syncwarp();
      if (lane == 0) mbar_arrive(&full[s]);
    }
    // db: the CTA's warps first, then one atomic per channel (atomics on one
    // address take about 40 ns each: with one per warp they were 0.1 ms of a
    // launch of 296 CTAs)
#pragma unroll
    for (int e = 0; e < 8; ++e) {
      float x = dbp[e];
      x += __shfl_xor_sync(0xffffffffu, x, 8);
      x += __shfl_xor_sync(0xffffffffu, x, 16);
      if (lane < 8) sdb[xw * 64 + o0 + e] = x;
    }
    asm volatile("bar.sync 1, %0;" ::"n"(32 * kBwdXWarps) : "memory");
    if (xt < 64 && !*abort_flag) {
      float x = 0.f;
#pragma unroll
      for (int w = 0; w < kBwdXWarps; ++w) x += sdb[w * 64 + xt];
      atomicAdd(p.db + xt, x);
    }
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  if (warp == 0) tmem_dealloc(tmem_base, kTmemCols);
}

// Backward of the projection head on tcgen05, per 128-pixel tile (h = Q1 v + b1):
//   h - b1 = v Q1^T                 (M 128 px, N 128 j, K 64 c)   GEMM-h
//   dh = dout Q2 GELU'(h), g = dout GELU(h)                        CUDA cores
//   dv = dh Q1                      (M 128 px, N 64 c,  K 128 j)  GEMM-dv
//   dQ1 += dh^T v                   (M 128 j,  N 64 c,  K 128 px) GEMM-Q
//   db1 += dh^T 1, dQ2 += g^T 1     (M 128 j,  N 16,    K 128 px)
//   db2 += sum dout.
// Warp 0 loads the v tile (TMA, 128B swizzle), warp 1 issues the MMAs (one
// thread), warps 2..9 (two per tensor-memory lane quadrant, each half of
// the columns) do the elementwise part, write the BF16 operands dh and g as
// rows of pixels (128B-swizzled boxes of 64 j) and drain dv.  The sums over
// pixels read dh, g and v MN-major, as they lie, and GEMM-dv reads Q1 the same
// way.  dv's accumulator takes h's columns.  The weight-gradient sums stay in
// tensor memory over all tiles of the CTA and are added to global memory once.
// Two CTAs per SM, persistent: one's GEMMs run under the other's elementwise
// part, which bounds it (erff and expf for 128 hidden units per pixel):
// 8 x 512^2: 0.87 -> 0.57 ms against one CTA with operands transposed by
// 2-byte stores and dv stored one pixel per lane.
constexpr int kPbThreads = 320;
constexpr uint32_t kPbQ1 = 0, kPbOnes = 16384, kPbV = 20480, kPbDH = 36864, kPbG = 69632, kPbOut = 102400,
                   kPbVec = 110592, kPbBars = 111616;
constexpr size_t kPbSmem = 1024 + kPbBars + 128;
static_assert(10 * 8 + 4 * 4 <= 128, "barriers, slot, flag and four sums");
static_assert(2 * (kPbSmem + 1024) <= 228 * 1024, "fno_tc_proj_bwd: two CTAs per SM");

struct FnoProjBwdParams {
  int tiles;
  const float* Q1;    // [128 j][64 c]
  const float* b1;    // [128]
  const float* q2;    // [128]
  const float* dout;  // [pix]
  float* dQ1;         // [128][64], accumulated
  float* db1;         // [128]
  float* dQ2;         // [128]
  float* db2;         // [1]
  int* err;
  unsigned long long probe_wait_ns;  // one warp's wait at the end runs out after this time (0: none)
};

__global__ void __launch_bounds__(kPbThreads, 2)
    fno_tc_proj_bwd(const __grid_constant__ CUtensorMap tmV, const __grid_constant__ CUtensorMap tmDv,
                    FnoProjBwdParams p) {
  extern __shared__ uint8_t smem_raw[];
  const uint32_t raw = smem_u32(smem_raw);
  uint8_t* base = smem_raw + (((raw + 1023u) & ~1023u) - raw);
  float* sb = reinterpret_cast<float*>(base + kPbVec);  // b1[128], Q2[128]
  uint64_t* bars = reinterpret_cast<uint64_t*>(base + kPbBars);
  uint64_t* v_full = bars + 0;
  uint64_t* h_full = bars + 1;
  uint64_t* ops_full = bars + 2; // 8 elementwise warps: h read, dh and g written
  uint64_t* dv_full = bars + 3;
  uint64_t* ops_free = bars + 4; // every MMA of the tile (v, dh, g are free)
  uint64_t* dv_free = bars + 5;  // 8 elementwise warps
  uint64_t* w_ready = bars + 6;  // 8 elementwise warps
  uint64_t* done = bars + 7;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 8);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
  float* sd2 = reinterpret_cast<float*>(tmem_slot + 2);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  constexpr uint32_t kTmemCols = 256;
  constexpr uint32_t cH = 0, cDV = 0, cQ = 128, cB = 192, cG = 208;  // accumulator columns

  if (threadIdx.x == 0) {
    mbar_init(v_full, 1);
    mbar_init(h_full, 1);
    mbar_init(ops_full, 8);
    mbar_init(dv_full, 1);
    mbar_init(ops_free, 1);
    mbar_init(dv_free, 8);
    mbar_init(w_ready, 8);
    mbar_init(done, 1);
    *abort_flag = 0;
    fence_barrier_init();
  }
  if (warp == 0) {
    tmem_alloc(tmem_slot, kTmemCols);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  auto fail = [&](int code) {
    *abort_flag = 1;
    if (p.err) atomicExch(p.err, code);
  };

  if (warp == 0) {
    if (lane == 0) {
      prefetch_tmap(&tmV);
      prefetch_tmap(&tmDv);
      int it = 0;
      for (int t = blockIdx.x; t < p.tiles && !*abort_flag; t += gridDim.x, ++it) {
        if (!mbar_wait_or_abort(ops_free, (it & 1) ^ 1, kFnoWaitNs, abort_flag)) {
          fail(41);
          break;
        }
        mbar_arrive_expect_tx(v_full, kTile);
        tma_load_2d(base + kPbV, &tmV, 0, t * 128, v_full);
      }
      // the last load issued lands before the CTA may exit
      if (it > 0) mbar_wait(v_full, (it - 1) & 1, kFnoWaitNs);
    }
  } else if (warp == 1) {
    if (lane == 0) {
      bool ok = mbar_wait_or_abort(w_ready, 0, kFnoWaitNs, abort_flag);
      if (!ok) fail(42);
      const uint32_t aV = smem_u32(base + kPbV), aQ = smem_u32(base + kPbQ1), aD = smem_u32(base + kPbDH),
                     aG = smem_u32(base + kPbG), aO = smem_u32(base + kPbOnes);
      int it = 0;
      for (int t = blockIdx.x; t < p.tiles && ok && !*abort_flag; t += gridDim.x, ++it) {
        const uint32_t ph = it & 1;
        if (!mbar_wait_or_abort(v_full, ph, kFnoWaitNs, abort_flag) ||
            !mbar_wait_or_abort(dv_free, ph ^ 1, kFnoWaitNs, abort_flag)) {
          fail(43);
          break;
        }
        tc_fence_after();
        {
          const uint64_t a = smem_desc_sw128(aV), b = smem_desc_sw128(aQ);
#pragma unroll
          for (int ks = 0; ks < 4; ++ks)
            tc_mma_bf16(tmem_base + cH, a + 2 * ks, b + 2 * ks, idesc_bf16(128, 128), ks > 0 ? 1u : 0u);
        }
        tc_commit(h_full);
        if (!mbar_wait_or_abort(ops_full, ph, kFnoWaitNs, abort_flag)) {
          fail(44);
          break;
        }
        tc_fence_after();
        const uint64_t qmn = smem_desc_sw128_mn(aQ, 16384), dmn = smem_desc_sw128_mn(aD, 16384),
                       gmn = smem_desc_sw128_mn(aG, 16384), vmn = smem_desc_sw128_mn(aV, 16384);
#pragma unroll
        for (int ks = 0; ks < 8; ++ks)
          tc_mma_bf16(tmem_base + cDV, smem_desc_sw128(aD + (ks >> 2) * 16384) + 2 * (ks & 3), qmn + kMnStep * ks,
                      idesc_bf16(128, 64) | kIdescBMn, ks > 0 ? 1u : 0u);
        tc_commit(dv_full);
#pragma unroll
        for (int ks = 0; ks < 8; ++ks) {
          const uint32_t acc = (it > 0 || ks > 0) ? 1u : 0u;
          const uint64_t one = smem_desc_sw128(aO + (ks >> 2) * 2048) + 2 * (ks & 3);
          tc_mma_bf16(tmem_base + cQ, dmn + kMnStep * ks, vmn + kMnStep * ks,
                      idesc_bf16(128, 64) | kIdescAMn | kIdescBMn, acc);
          tc_mma_bf16(tmem_base + cB, dmn + kMnStep * ks, one, idesc_bf16(128, 16) | kIdescAMn, acc);
          tc_mma_bf16(tmem_base + cG, gmn + kMnStep * ks, one, idesc_bf16(128, 16) | kIdescAMn, acc);
        }
        tc_commit(ops_free);
      }
      tc_commit(done);
      mbar_wait(done, 0, kFnoWaitNs);
    }
  } else {
    // elementwise warps 2..9: lane quadrant warp % 4 (pixel rows of a tile,
    // j rows of the weight-gradient sums), column half `half`
    const int quad = warp & 3, half = (warp - 2) >> 2;
    const int et = threadIdx.x - 64;  // 0..255
    // resident operands: Q1 [j][c] and ones (row 0 of 16)
    for (int e = et; e < 128 * 64; e += 256) {
      const int j = e >> 6, c = e & 63;
      *reinterpret_cast<__nv_bfloat16*>(base + kPbQ1 + sw128_off(j, c)) = __float2bfloat16_rn(p.Q1[e]);
    }
    for (int e = et; e < 2 * 16 * 64; e += 256) {
      const int bx = e >> 10, r = (e >> 6) & 15, k = e & 63;
      *reinterpret_cast<__nv_bfloat16*>(base + kPbOnes + bx * 2048 + sw128_off(r, k)) =
          __float2bfloat16_rn(r == 0 ? 1.f : 0.f);
    }
    sb[et] = et < 128 ? p.b1[et] : p.q2[et - 128];
    fence_proxy_async_smem();
    asm volatile("bar.sync 1, 256;" ::: "memory");  // sb is read by every elementwise warp
    if (lane == 0) mbar_arrive(w_ready);

    const int px = quad * 32 + lane;  // pixel row within the tile
    const uint32_t lrow = static_cast<uint32_t>(quad * 32) << 16;
    uint8_t* so = base + kPbOut + (warp - 2) * 1024;  // dv staging: 32 px x 8 channels
    float gd2 = 0.f;
    int it = 0, nst = 0;
    for (int t = blockIdx.x; t < p.tiles; t += gridDim.x, ++it) {
      const uint32_t ph = it & 1;
      const float d = p.dout[static_cast<size_t>(t) * 128 + px];
      const bool ok = __all_sync(0xffffffffu, mbar_wait_or_abort(h_full, ph, kFnoWaitNs, abort_flag) &&
                                                  mbar_wait_or_abort(ops_free, ph ^ 1, kFnoWaitNs, abort_flag));
      if (!ok) {
        if (lane == 0) fail(45);
        break;
      }
      tc_fence_after();
      if (half == 0) gd2 += d;
#pragma unroll 1
      for (int jc = 0; jc < 2; ++jc) {
        const int j0 = half * 64 + jc * 32;
        float h[32];
        tmem_ld32(tmem_base + lrow + cH + j0, h);
        uint8_t* dbox = base + kPbDH + half * 16384;
        uint8_t* gbox = base + kPbG + half * 16384;
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          uint32_t dw[4], gw[4];
#pragma unroll
          for (int i = 0; i < 8; i += 2) {
            float dh[2], gg[2];
            const float2 bj = *reinterpret_cast<const float2*>(sb + j0 + 8 * q + i);
            const float2 qj = *reinterpret_cast<const float2*>(sb + 128 + j0 + 8 * q + i);
#pragma unroll
            for (int k = 0; k < 2; ++k) {
              const float x = h[8 * q + i + k] + (k ? bj.y : bj.x);
              const float cdf = 0.5f * (1.f + erff(x * 0.70710678118654752f));
              const float pdf = 0.39894228040143268f * expf(-0.5f * x * x);
              dh[k] = d * (k ? qj.y : qj.x) * (cdf + x * pdf);
              gg[k] = d * x * cdf;
            }
            const __nv_bfloat162 db2 = __floats2bfloat162_rn(dh[0], dh[1]), gb2 = __floats2bfloat162_rn(gg[0], gg[1]);
            dw[i / 2] = *reinterpret_cast<const uint32_t*>(&db2);
            gw[i / 2] = *reinterpret_cast<const uint32_t*>(&gb2);
          }
          const uint32_t o = sw128_off(px, jc * 32 + 8 * q);
          *reinterpret_cast<uint4*>(dbox + o) = make_uint4(dw[0], dw[1], dw[2], dw[3]);
          *reinterpret_cast<uint4*>(gbox + o) = make_uint4(gw[0], gw[1], gw[2], gw[3]);
        }
      }
      fence_proxy_async_smem();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(ops_full);
      // dv: this half's 32 channels of pixel row px
      const bool got = __all_sync(0xffffffffu, mbar_wait_or_abort(dv_full, ph, kFnoWaitNs, abort_flag));
      if (!got) {
        if (lane == 0) fail(46);
        break;
      }
      tc_fence_after();
      float o[32];
      tmem_ld32(tmem_base + lrow + cDV + half * 32, o);
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(dv_free);
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        if (lane == 0 && nst > 0) bulk_wait_read<0>();
        __syncwarp();
        float4* w = reinterpret_cast<float4*>(so + lane * 32);
        w[0] = make_float4(o[8 * q], o[8 * q + 1], o[8 * q + 2], o[8 * q + 3]);
        w[1] = make_float4(o[8 * q + 4], o[8 * q + 5], o[8 * q + 6], o[8 * q + 7]);
        fence_proxy_async_smem();
        __syncwarp();
        if (lane == 0) {
          tma_store_2d(&tmDv, so, half * 32 + 8 * q, t * 128 + quad * 32);
          bulk_commit();
        }
        ++nst;
      }
    }
    // every TMA store must have finished before the CTA's shared memory goes
    if (lane == 0 && nst > 0) bulk_wait<0>();
    __syncwarp();
    // weight-gradient sums: rows j = lanes of the quadrant.  Whether they are
    // added is each warp's own finding (its wait, or the flag of another's):
    // the barrier of the db2 sum lies outside, where every warp comes by.
    const bool fin = __all_sync(0xffffffffu, mbar_wait(done, 0, kFnoWaitNs) &&
                                                 (!p.probe_wait_ns || half != 0 || quad != 1 ||
                                                  mbar_wait(done, 1, p.probe_wait_ns)));  // no second phase comes
    const bool add = __all_sync(0xffffffffu, fin && !*abort_flag);
    if (half == 0) {
#pragma unroll
      for (int sh = 16; sh > 0; sh >>= 1) gd2 += __shfl_xor_sync(0xffffffffu, gd2, sh);
      if (lane == 0) sd2[quad] = gd2;
      asm volatile("bar.sync 2, 128;" ::: "memory");
      if (add && quad == 0 && lane == 0) atomicAdd(p.db2, (sd2[0] + sd2[1]) + (sd2[2] + sd2[3]));
    }
    if (add) {
      tc_fence_after();
      const int j = quad * 32 + lane;
      float a[32];
      tmem_ld32(tmem_base + lrow + cQ + half * 32, a);
      // eight columns at a time through the staging tile: whole sectors per atomic
      float* sf = reinterpret_cast<float*>(so);
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        __syncwarp();
        *reinterpret_cast<float4*>(sf + lane * 8) = make_float4(a[8 * q], a[8 * q + 1], a[8 * q + 2], a[8 * q + 3]);
        *reinterpret_cast<float4*>(sf + lane * 8 + 4) = make_float4(a[8 * q + 4], a[8 * q + 5], a[8 * q + 6], a[8 * q + 7]);
        __syncwarp();
#pragma unroll
        for (int r = 0; r < 8; ++r)
          atomicAdd(p.dQ1 + (quad * 32 + 4 * r + (lane >> 3)) * 64 + half * 32 + 8 * q + (lane & 7), sf[32 * r + lane]);
      }
      if (half == 0) {
        float b[16], g[16];
        tmem_ld16(tmem_base + lrow + cB, b);
        tmem_ld16(tmem_base + lrow + cG, g);
        atomicAdd(p.db1 + j, b[0]);
        atomicAdd(p.dQ2 + j, g[0]);
      }
    } else if (!fin && lane == 0) {
      fail(47);
    }
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  if (warp == 0) tmem_dealloc(tmem_base, kTmemCols);
}

// bf16 copies of a forward's weights, one launch for all of them (one per
// matrix before): the layers' matrices W (n values each, `stride` apart) into
// wb, then Q1 (nq values) into q1b.  grid: (blocks, layers + 1).
__global__ void __launch_bounds__(256) fno_to_bf16(const float* __restrict__ W, size_t stride, int layers, int n,
                                                    __nv_bfloat16* __restrict__ wb, const float* __restrict__ Q1, int nq,
                                                    __nv_bfloat16* __restrict__ q1b) {
  const int l = blockIdx.y;
  const float* a = l < layers ? W + l * stride : Q1;
  __nv_bfloat16* b = l < layers ? wb + static_cast<size_t>(l) * n : q1b;
  const int m = l < layers ? n : nq;
  for (int i = blockIdx.x * 256 + threadIdx.x; i < m; i += gridDim.x * 256) b[i] = __float2bfloat16_rn(a[i]);
}

// Tw[x][kk] (bf16, kk < 32): cos / sin of 2 pi kx x / S for kk = 2 kx / 2 kx + 1
// < 2m, zero beyond; from twx[kx][x] = (cos, -sin).
__global__ void fno_tw_table(const float2* __restrict__ twx, int S, int m, __nv_bfloat16* __restrict__ Tw) {
  for (int t = blockIdx.x * blockDim.x + threadIdx.x; t < S * 32; t += gridDim.x * blockDim.x) {
    const int kk = t & 31, x = t >> 5;
    float v = 0.f;
    if (kk < 2 * m) {
      const float2 w = twx[static_cast<size_t>(kk >> 1) * S + x];
      v = (kk & 1) ? -w.y : w.x;
    }
    Tw[t] = __float2bfloat16_rn(v);
  }
}

}  // namespace huv_dev

namespace huv_launch {
unsigned long long probe_wait_ns();
bool tc_map_bf16(CUtensorMap* map, const void* ptr, uint64_t rows, int kp, int box_rows);

bool tc_map_out(CUtensorMap* map, void* ptr, uint64_t rows, uint64_t cols);
bool tc_map_out8(CUtensorMap* map, void* ptr, uint64_t rows, uint64_t cols);
bool tc_map_sw64_bf16(CUtensorMap* map, const void* ptr, uint64_t rows, int kp, int box_rows, int cols);

cudaError_t fno_tc_set_smem() {
  cudaError_t e;
  if ((e = cudaFuncSetAttribute(huv_dev::fno_tc_layer, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                static_cast<int>(huv_dev::kFnoLayerSmem))))
    return e;
  if ((e = cudaFuncSetAttribute(huv_dev::fno_tc_layer_bwd, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                static_cast<int>(huv_dev::kBwdSmem))))
    return e;
  if ((e = cudaFuncSetAttribute(huv_dev::fno_tc_proj_bwd, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                static_cast<int>(huv_dev::kPbSmem))))
    return e;
  return cudaFuncSetAttribute(huv_dev::fno_tc_proj, cudaFuncAttributeMaxDynamicSharedMemorySize,
                              static_cast<int>(huv_dev::kFnoProjSmem));
}

// Layer l forward on tensor cores.  v: [B*S*S][64] bf16; Wb: [64][64] bf16;
// Tw: [S][32] bf16; Zs: [B*S*64][32] bf16; zsave may be null.
bool fno_tc_layer(int B, int S, int m, const __nv_bfloat16* v, const __nv_bfloat16* Wb,
                  const __nv_bfloat16* Tw, const __nv_bfloat16* Zs, const float* bias, int act,
                  __nv_bfloat16* zsave, __nv_bfloat16* vnext, int* err, cudaStream_t st) {
  CUtensorMap mv, mw, mt, mz, mvn, mzo;
  const uint64_t pix = static_cast<uint64_t>(B) * S * S;
  if (!tc_map_bf16(&mv, v, pix, 64, 128) || !tc_map_bf16(&mw, Wb, 64, 64, 64) ||
      !tc_map_sw64_bf16(&mt, Tw, static_cast<uint64_t>(S), 32, 128, 32) ||
      !tc_map_sw64_bf16(&mz, Zs, static_cast<uint64_t>(B) * S * 64, 32, 64, 32) ||
      !tc_map_sw64_bf16(&mvn, vnext, pix, 64, 32, 64) || !tc_map_sw64_bf16(&mzo, zsave ? zsave : vnext, pix, 64, 32, 64))
    return false;
  huv_dev::FnoTcParams p{};
  p.tiles = static_cast<int>(pix / 128);
  p.S = S;
  p.kk_steps = (2 * m + 15) / 16;
  p.bias = bias;
  p.act = act;
  p.save_z = zsave ? 1 : 0;
  p.err = err;
  const int grid = std::min(p.tiles, 2 * 148);
  huv_dev::fno_tc_layer<<<grid, 32 * (2 + huv_dev::kFnoEpiWarps), huv_dev::kFnoLayerSmem, st>>>(mv, mw, mt, mz, mvn,
                                                                                               mzo, p);
  return cudaGetLastError() == cudaSuccess;
}

// Projection head on tensor cores.  Q1b: [128][64] bf16.
bool fno_tc_proj(int B, int S, const __nv_bfloat16* v, const __nv_bfloat16* Q1b, const float* b1, const float* q2,
                 const float* b2, float* out, int* err, cudaStream_t st) {
  CUtensorMap mv, mq;
  const uint64_t pix = static_cast<uint64_t>(B) * S * S;
  if (!tc_map_bf16(&mv, v, pix, 64, 128) || !tc_map_bf16(&mq, Q1b, 128, 64, 128)) return false;
  huv_dev::FnoTcParams p{};
  p.tiles = static_cast<int>(pix / 128);
  p.S = S;
  p.bias = b1;
  p.q2 = q2;
  p.b2 = b2;
  p.out = out;
  p.err = err;
  const int grid = std::min(p.tiles, 2 * 148);
  huv_dev::fno_tc_proj<<<grid, 32 * (2 + huv_dev::kFnoEpiWarps), huv_dev::kFnoProjSmem, st>>>(mv, mq, p);
  return cudaGetLastError() == cudaSuccess;
}
// Layer backward on tensor cores (see fno_tc_layer_bwd); pix a multiple of 128.
bool fno_tc_layer_bwd(size_t pix, const float* dvnext, const __nv_bfloat16* z, const __nv_bfloat16* v, const float* W,
                      int act, float* dz, float* dv, float* dW, float* db, int* err, cudaStream_t st) {
  if (pix % 128 != 0) return false;
  CUtensorMap mv, mo;
  if (!tc_map_bf16(&mv, v, pix, 64, 128) || !tc_map_out(&mo, dv, pix, 64)) return false;
  huv_dev::FnoBwdParams p{};
  p.tiles = static_cast<int>(pix / 128);
  p.act = act;
  p.dvnext = dvnext;
  p.z = z;
  p.W = W;
  p.dz = dz;
  p.dW = dW;
  p.db = db;
  p.err = err;
  int sms = 0, dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess)
    return false;
  const int grid = std::min(p.tiles, 2 * sms);
  huv_dev::fno_tc_layer_bwd<<<grid, huv_dev::kBwdThreads, huv_dev::kBwdSmem, st>>>(mv, mo, p);
  return cudaGetLastError() == cudaSuccess;
}
// Projection backward on tensor cores (see fno_tc_proj_bwd); v: [pix][64]
// bf16, pix a multiple of 128.
bool fno_tc_proj_bwd(size_t pix, const __nv_bfloat16* v, const float* Q1, const float* b1, const float* q2,
                     const float* dout, float* dv, float* dQ1, float* db1, float* dQ2, float* db2, int* err,
                     cudaStream_t st) {
  if (pix % 128 != 0) return false;
  CUtensorMap mv, mo;
  if (!tc_map_bf16(&mv, v, pix, 64, 128) || !tc_map_out8(&mo, dv, pix, 64)) return false;
  huv_dev::FnoProjBwdParams p{};
  p.tiles = static_cast<int>(pix / 128);
  p.Q1 = Q1;
  p.b1 = b1;
  p.q2 = q2;
  p.dout = dout;
  p.dQ1 = dQ1;
  p.db1 = db1;
  p.dQ2 = dQ2;
  p.db2 = db2;
  p.err = err;
  p.probe_wait_ns = probe_wait_ns();
  int sms = 0, dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess)
    return false;
  const int grid = std::min(p.tiles, 2 * sms);
  huv_dev::fno_tc_proj_bwd<<<grid, huv_dev::kPbThreads, huv_dev::kPbSmem, st>>>(mv, mo, p);
  return cudaGetLastError() == cudaSuccess;
}
void fno_tc_weights(const float* W, size_t stride, int layers, int n, __nv_bfloat16* wb, const float* Q1, int nq,
                    __nv_bfloat16* q1b, cudaStream_t st) {
  huv_dev::fno_to_bf16<<<dim3(8, layers + 1), 256, 0, st>>>(W, stride, layers, n, wb, Q1, nq, q1b);
}
void fno_tc_tw_table(const float2* twx, int S, int m, __nv_bfloat16* Tw, cudaStream_t st) {
  huv_dev::fno_tw_table<<<(S * 32 + 255) / 256, 256, 0, st>>>(twx, S, m, Tw);
}
}  // namespace huv_launch
