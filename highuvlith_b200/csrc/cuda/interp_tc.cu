// Separable band interpolation I_N = P I_M P^T in one tcgen05 kernel, for
// evaluation grids M that are multiples of 16 up to 160 and output grids N
// that are multiples of 256.
//
// P is the real N x M Dirichlet matrix of the band |f| <= 2h < M / 2
// (Engine::interp_matrix) as FP16 hi/lo planes; the coarse image I_M arrives
// as FP16 hi/lo planes divided by interp_scale(mean).  One CTA per (clip, 256
// output columns X) does both products:
//   1. Z^T(X, y) = sum_x P(X, x) I_M(y, x): two 128-row accumulators of M
//      columns, I_M's planes resident in shared memory, P's rows streamed;
//   2. the epilogue warps split Z^T into FP16 hi/lo and write it, as the
//      K-major B operand of the second product, over I_M's bytes;
//   3. I_N(Y, X) = sum_y P(Y, y) Z^T(X, y) for every 128-row tile Y, P's rows
//      streamed, 128 x 256 accumulators double-buffered in tensor memory,
//      the epilogue multiplying interp_scale back and storing with TMA.
// Every product is hi.hi + hi.lo + lo.hi with FP32 accumulation.
//
// What bounds it: the latency of P's stream and the set-up of a CTA (I_M, the
// first product and its split: a fifth of its time).  Z^T stays on chip and an
// output tile streams P's 80 KB from L2, in contiguous 8 KB copies of the
// tiled operand, where the two-kernel path wrote Z^T to HBM and streamed
// 160 KB of it back per tile.  256 clips of 1024^2 at M = 160: 0.382 -> 0.300 ms
// (3.6 TB/s of image).  On the way: four epilogue warps with 4 KB tiles, P by
// tensor copies of 64-byte rows, 4 stages 0.367, 6 stages 0.317; eight warps
// with 2 KB tiles 0.308; contiguous copies 0.300 (0.349 with 4 stages).  With a
// third of the products 0.266, without stores 0.291, with neither 0.232;
// 256-bit stores from registers 0.375.
#include <cuda.h>
#include <cuda_fp16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include "../engine.hpp"
#include "fft_reg.cuh"
#include "tc_ptx.cuh"

namespace huv_dev {

constexpr int kIfMaxM = 160;
constexpr uint32_t kIfPBox = 128 * 64;    // 128 rows of P x 32 fp16, one plane
constexpr uint32_t kIfZBox = 256 * 64;    // 256 rows X of Z^T x 32 fp16, one plane
constexpr uint32_t kIfOutTile = 32 * 16 * 4;  // 32 rows Y x 16 columns X
constexpr int kIfEpiWarps = 8;            // two per tensor-memory lane quadrant
// staging tiles per epilogue warp: one where Z^T leaves little room for P's
// stages, of which the kernel wants many
__host__ __device__ constexpr int if_out_bufs(int M) { return M > 96 ? 1 : 2; }
constexpr int kIfMaxStages = 10;
constexpr uint64_t kIfWaitNs = 2000000000ull;

__host__ __device__ constexpr int if_boxes(int M) { return (M + 31) / 32; }
__host__ __device__ constexpr size_t if_fixed_bytes(int M) {
  return 1024 + 2 * static_cast<size_t>(if_boxes(M)) * kIfZBox + kIfEpiWarps * if_out_bufs(M) * static_cast<size_t>(kIfOutTile) + 256;
}
// P stages of 8 KB: what one CTA's shared memory holds beside Z^T (6 at M = 160)
__host__ __device__ constexpr int if_stages(int M) {
  const int s = static_cast<int>((232448 - if_fixed_bytes(M)) / kIfPBox);
  return s > kIfMaxStages ? kIfMaxStages : s;
}
__host__ __device__ constexpr size_t if_smem_bytes(int M) {
  return if_fixed_bytes(M) + static_cast<size_t>(if_stages(M)) * kIfPBox;
}
static_assert(if_stages(kIfMaxM) >= 6 && if_smem_bytes(kIfMaxM) <= 232448, "tc_interp_fused: shared memory");

struct InterpParams {
  int M, stages;
  int n;               // output grid side (rows of P per plane)
  int mt, mt_per;      // 128-row output tiles, and tiles per CTA
  const uint8_t* P;    // [row tile][box][plane] x 8 KB, 64B-swizzled
  const float* mean;
  int* err;
  unsigned long long probe_wait_ns;
};

template <int OUTBUFS>
__global__ void __launch_bounds__(32 * (2 + kIfEpiWarps), 1)
    tc_interp_fused(const __grid_constant__ CUtensorMap tmI, const __grid_constant__ CUtensorMap tmO, InterpParams p) {
  extern __shared__ uint8_t smem_raw[];
  const uint32_t raw = smem_u32(smem_raw);
  uint8_t* base = smem_raw + (((raw + 1023u) & ~1023u) - raw);
  const int nbox = if_boxes(p.M), ksteps = p.M / 16;
  uint8_t* sZ = base;                               // [plane][box] Z^T; first [plane][box] I_M
  uint8_t* sP = sZ + 2 * nbox * kIfZBox;            // [stage] one plane, one box
  uint8_t* sO = sP + p.stages * kIfPBox;            // [epilogue warp][buffer]
  uint64_t* bars = reinterpret_cast<uint64_t*>(sO + kIfEpiWarps * OUTBUFS * kIfOutTile);
  uint64_t* full = bars;
  uint64_t* empty = bars + kIfMaxStages;
  uint64_t* i_full = bars + 2 * kIfMaxStages;
  uint64_t* z_full = i_full + 1;   // stage-1 accumulators complete
  uint64_t* z_ready = i_full + 2;  // Z^T planes written (one arrival per epilogue warp)
  uint64_t* tfull = i_full + 3;
  uint64_t* tempty = i_full + 5;
  uint64_t* done = i_full + 7;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(i_full + 8);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int xt = blockIdx.x, prob = blockIdx.z;
  const int m0 = blockIdx.y * p.mt_per, m1 = min(p.mt, m0 + p.mt_per);
  const uint32_t ibox = static_cast<uint32_t>(p.M) * 64;  // M rows y x 32 fp16

  if (threadIdx.x == 0) {
    for (int s = 0; s < p.stages; ++s) {
      mbar_init(&full[s], 1);
      mbar_init(&empty[s], 1);
    }
    mbar_init(i_full, 1);
    mbar_init(z_full, 1);
    mbar_init(z_ready, kIfEpiWarps);
    mbar_init(&tfull[0], 1);
    mbar_init(&tfull[1], 1);
    mbar_init(&tempty[0], kIfEpiWarps);
    mbar_init(&tempty[1], kIfEpiWarps);
    mbar_init(done, 1);
    *abort_flag = 0;
    fence_barrier_init();
  }
  if (warp == 0) {
    tmem_alloc(tmem_slot, 512);
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
      prefetch_tmap(&tmI);
      prefetch_tmap(&tmO);
      mbar_arrive_expect_tx(i_full, 2u * nbox * ibox);
      for (int pl = 0; pl < 2; ++pl)
        for (int kb = 0; kb < nbox; ++kb)
          tma_load_2d(sZ + (pl * nbox + kb) * ibox, &tmI, kb * 32, (prob * 2 + pl) * p.M, i_full);
      // P rows: the CTA's 256 columns X (two tiles), then its output rows Y
      int it = 0;
      bool ok = true;
      const int tiles = 2 + m1 - m0;
      for (int t = 0; t < tiles && ok && !*abort_flag; ++t) {
        // the row tile's boxes are contiguous: [box][plane] x 8 KB
        const uint8_t* src = p.P + static_cast<size_t>(t < 2 ? xt * 2 + t : m0 + t - 2) * 2 * nbox * kIfPBox;
        for (int kb = 0; kb < nbox && ok; ++kb)
          for (int pl = 0; pl < 2; ++pl, ++it) {
            const int s = it % p.stages;
            if (!mbar_wait_or_abort(&empty[s], ((it / p.stages) & 1) ^ 1, kIfWaitNs, abort_flag)) {
              fail(51);
              ok = false;
              break;
            }
            mbar_arrive_expect_tx(&full[s], kIfPBox);
            bulk_load(sP + s * kIfPBox, src + (kb * 2 + pl) * kIfPBox, kIfPBox, &full[s]);
          }
      }
      // every load issued must have landed before the CTA may exit
      mbar_wait(i_full, 0, kIfWaitNs);
      for (int q = (it > p.stages ? it - p.stages : 0); q < it; ++q)
        mbar_wait(&full[q % p.stages], (q / p.stages) & 1, kIfWaitNs);
    }
  } else if (warp == 1) {
    if (lane == 0) {
      bool ok = mbar_wait(i_full, 0, kIfWaitNs);
      if (!ok) fail(52);
      if (ok && p.probe_wait_ns && !mbar_wait(done, 0, p.probe_wait_ns)) {  // nothing arrives at `done` yet
        fail(56);
        ok = false;
      }
      tc_fence_after();
      int it = 0;
      // one 128-row tile of P against the resident operand at `b` (its planes
      // `bplane` bytes apart, its boxes `bbox`), into the accumulator at d;
      // both planes of a box are taken together.  The order of the split
      // products is the two-kernel path's (tc_dft_gemm<3>, tc_interp_w256), so
      // that an image has the same bits whichever of them made it.
      auto tile = [&](uint32_t d, uint32_t b, uint32_t bplane, uint32_t bbox, uint32_t idesc,
                      bool second) {
        for (int kb = 0; kb < nbox; ++kb, it += 2) {
          const int s0 = it % p.stages, s1 = (it + 1) % p.stages;
          if (!mbar_wait(&full[s0], (it / p.stages) & 1, kIfWaitNs) ||
              !mbar_wait(&full[s1], ((it + 1) / p.stages) & 1, kIfWaitNs)) {
            fail(54);
            return false;
          }
          tc_fence_after();
          const uint64_t ah = smem_desc_sw64(smem_u32(sP + s0 * kIfPBox)), al = smem_desc_sw64(smem_u32(sP + s1 * kIfPBox));
          const uint64_t bh = smem_desc_sw64(b + kb * bbox), bl = smem_desc_sw64(b + bplane + kb * bbox);
#pragma unroll
          for (int ks = 0; ks < 2; ++ks) {
            const uint64_t adv = static_cast<uint64_t>(2 * ks);  // 32 bytes per 16-wide K step
            if (kb * 2 + ks < ksteps) {
              tc_mma_bf16(d, ah + adv, bh + adv, idesc, kb + ks > 0 ? 1u : 0u);
              if (!second) tc_mma_bf16(d, ah + adv, bl + adv, idesc, 1u);
              tc_mma_bf16(d, al + adv, bh + adv, idesc, 1u);
            }
          }
          if (second)
#pragma unroll
            for (int ks = 0; ks < 2; ++ks) {
              const uint64_t adv = static_cast<uint64_t>(2 * ks);
              if (kb * 2 + ks < ksteps) tc_mma_bf16(d, ah + adv, bl + adv, idesc, 1u);
            }
          tc_commit(&empty[s0]);
          tc_commit(&empty[s1]);
        }
        return true;
      };
      const uint32_t zaddr = smem_u32(sZ);
      for (int t = 0; t < 2 && ok; ++t)
        ok = tile(tmem_base + t * 256, zaddr, nbox * ibox, ibox, idesc_f16(128, p.M), false);
      if (ok) tc_commit(z_full);
      if (ok && !mbar_wait_or_abort(z_ready, 0, kIfWaitNs, abort_flag)) {
        fail(57);
        ok = false;
      }
      tc_fence_after();
      for (int i = 0; i < m1 - m0 && ok && !*abort_flag; ++i) {
        const int buf = i & 1;
        if (!mbar_wait_or_abort(&tempty[buf], ((i >> 1) & 1) ^ 1, kIfWaitNs, abort_flag)) {
          fail(53);
          break;
        }
        tc_fence_after();
        ok = tile(tmem_base + buf * 256, zaddr, nbox * kIfZBox, kIfZBox, idesc_f16(128, 256), true);
        if (ok) tc_commit(&tfull[buf]);
      }
      // all MMAs issued by this thread have completed once `done` flips
      tc_commit(done);
      mbar_wait(done, 0, kIfWaitNs);
    }
  } else {
    // epilogue warps 2..9: tensor-memory lane quadrant = warp % 4; warps 2..5
    // take the first tile of Z^T and half of an output tile's columns, 6..9 the second
    const int quad = warp & 3;
    const uint32_t lrow = tmem_base + (static_cast<uint32_t>(quad * 32) << 16);
    int nst = 0;  // TMA-store tiles issued by this warp
    bool got = __all_sync(0xffffffffu, mbar_wait_or_abort(z_full, 0, kIfWaitNs, abort_flag));
    if (got) {
      tc_fence_after();
      // Z^T -> FP16 hi/lo planes: row X of a box holds 32 y in four 16-byte
      // chunks (64B swizzle: chunk ^ (row / 2) % 4)
      {
        const int t = warp >= 6;
        const int row = t * 128 + quad * 32 + lane;
        const uint32_t sw = static_cast<uint32_t>(row >> 1) & 3u;
#pragma unroll 1
        for (int c0 = 0; c0 < p.M; c0 += 16) {
          float v[16];
          tmem_ld16(lrow + t * 256 + c0, v);
          uint32_t hw[8], lw[8];
#pragma unroll
          for (int i = 0; i < 8; ++i) {
            const __half2 h2 = __floats2half2_rn(v[2 * i], v[2 * i + 1]);
            const float2 hf = __half22float2(h2);
            const __half2 l2 = __floats2half2_rn(v[2 * i] - hf.x, v[2 * i + 1] - hf.y);
            hw[i] = *reinterpret_cast<const uint32_t*>(&h2);
            lw[i] = *reinterpret_cast<const uint32_t*>(&l2);
          }
          uint8_t* zh = sZ + (c0 >> 5) * kIfZBox + row * 64;
          uint8_t* zl = zh + nbox * kIfZBox;
          const uint32_t ch = static_cast<uint32_t>(c0 & 31) >> 3;
#pragma unroll
          for (int q = 0; q < 2; ++q) {
            const uint32_t o = ((ch + q) ^ sw) << 4;
            *reinterpret_cast<uint4*>(zh + o) = make_uint4(hw[4 * q], hw[4 * q + 1], hw[4 * q + 2], hw[4 * q + 3]);
            *reinterpret_cast<uint4*>(zl + o) = make_uint4(lw[4 * q], lw[4 * q + 1], lw[4 * q + 2], lw[4 * q + 3]);
          }
        }
      }
      fence_proxy_async_smem();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(z_ready);
    } else if (lane == 0) {
      fail(58);
    }
    const float osc = interp_scale(p.mean[prob]);
    for (int i = 0; i < m1 - m0 && got; ++i) {
      const int buf = i & 1;
      // warp-uniform outcome: tcgen05.ld below is .sync.aligned
      got = __all_sync(0xffffffffu, mbar_wait_or_abort(&tfull[buf], (i >> 1) & 1, kIfWaitNs, abort_flag));
      if (!got) {
        if (lane == 0) fail(55);
        break;
      }
      tc_fence_after();
#pragma unroll 1
      for (int c0 = (warp >= 6 ? 128 : 0); c0 < (warp >= 6 ? 256 : 128); c0 += 32) {
        float v[32];
        tmem_ld32(lrow + buf * 256 + c0, v);
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          if (lane == 0 && nst >= OUTBUFS) bulk_wait_read<OUTBUFS - 1>();
          __syncwarp();
          uint8_t* sb = sO + ((warp - 2) * OUTBUFS + nst % OUTBUFS) * kIfOutTile;
#pragma unroll
          for (int q = 0; q < 4; ++q)
            *reinterpret_cast<float4*>(sb + lane * 64 + ((q ^ ((lane >> 1) & 3)) << 4)) =
                make_float4(osc * v[16 * h + 4 * q], osc * v[16 * h + 4 * q + 1], osc * v[16 * h + 4 * q + 2], osc * v[16 * h + 4 * q + 3]);
          fence_proxy_async_smem();
          __syncwarp();
          if (lane == 0) {
            tma_store_2d(&tmO, sb, xt * 256 + c0 + 16 * h, prob * p.n + (m0 + i) * 128 + quad * 32);
            bulk_commit();
          }
          ++nst;
        }
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&tempty[buf]);
    }
    // every TMA store must have finished before the CTA's shared memory goes
    if (lane == 0 && nst > 0) bulk_wait<0>();
    __syncwarp();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  if (warp == 0) tmem_dealloc(tmem_base, 512);
}

}  // namespace huv_dev

namespace huv_launch {

bool tc_map_sw64_f16(CUtensorMap* map, const void* ptr, uint64_t rows, int kp, int box_rows, int cols);
bool tc_map_out16(CUtensorMap* map, void* ptr, uint64_t rows, uint64_t cols);
unsigned long long probe_wait_ns();

// Whether one kernel does the whole separable interpolation from M to n.
bool interp_fused_ok(int M, int n) { return M % 16 == 0 && M >= 16 && M <= huv_dev::kIfMaxM && n % 256 == 0 && M < n; }

// Byte offset of P's element (row, column) of plane pl in the tiled operand
// that the kernel streams, and the operand's size.
size_t interp_tiled_offset(int row, int col, int pl, int M) {
  const int nbox = huv_dev::if_boxes(M), r = row % 128, c = col % 32;
  return ((static_cast<size_t>(row / 128) * nbox + col / 32) * 2 + pl) * huv_dev::kIfPBox + r * 64 +
         ((c / 8) ^ ((r / 2) & 3)) * 16 + (c % 8) * 2;
}
size_t interp_tiled_bytes(int M, int n) {
  return static_cast<size_t>(n / 128) * huv_dev::if_boxes(M) * 2 * huv_dev::kIfPBox;
}

// Images of nc clips: P as tiled by interp_tiled_offset, I_M /
// interp_scale(mean) as FP16 planes [nc][2][M][M].
cudaError_t interp_fused(const void* P, const void* im_split, int M, int n, int nc, const float* mean,
                         float* out, int* err, cudaStream_t st) {
  static std::atomic<uint64_t> smem_set{0};
  huv::once_per_device(smem_set, [] {
    for (auto k : {huv_dev::tc_interp_fused<1>, huv_dev::tc_interp_fused<2>})
      huv::check_cuda(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, 232448),
                      "cudaFuncSetAttribute(interp)");
  });
  CUtensorMap mi, mo;
  if (!tc_map_sw64_f16(&mi, im_split, static_cast<uint64_t>(nc) * 2 * M, M, M, M) ||
      !tc_map_out16(&mo, out, static_cast<uint64_t>(nc) * n, n))
    return cudaErrorInvalidValue;
  int sms = 0, dev = 0;
  cudaError_t e;
  if ((e = cudaGetDevice(&dev)) != cudaSuccess) return e;
  if ((e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev)) != cudaSuccess) return e;
  huv_dev::InterpParams p{};
  p.M = M;
  p.stages = huv_dev::if_stages(M);
  p.n = n;
  p.mt = n / 128;
  // Few clips: the row tiles are split over more CTAs (each repeats the first
  // product) until one wave is full.
  int split = 1;
  while (split < p.mt && static_cast<long long>(n / 256) * split * 2 * nc <= sms) split *= 2;
  p.mt_per = (p.mt + split - 1) / split;
  p.P = static_cast<const uint8_t*>(P);
  p.mean = mean;
  p.err = err;
  p.probe_wait_ns = probe_wait_ns();
  const dim3 g(n / 256, (p.mt + p.mt_per - 1) / p.mt_per, nc);
  if (huv_dev::if_out_bufs(M) == 1)
    huv_dev::tc_interp_fused<1><<<g, 32 * (2 + huv_dev::kIfEpiWarps), huv_dev::if_smem_bytes(M), st>>>(mi, mo, p);
  else
    huv_dev::tc_interp_fused<2><<<g, 32 * (2 + huv_dev::kIfEpiWarps), huv_dev::if_smem_bytes(M), st>>>(mi, mo, p);
  return cudaGetLastError();
}

}  // namespace huv_launch
