// Programmatic dependent launch: a kernel's blocks may be placed, and its
// launch processed, while the kernel before it on the stream still runs.
//
// Every kernel launched with `pdl` starts with pdl_begin(): it lets the next
// kernel be placed once all of its own blocks have started, then waits until
// everything before it on the stream has completed and its writes are
// visible.  Nothing is read, written or returned before that, so the order of
// memory operations is that of plain launches; what overlaps is launch
// latency (a chain of small kernels: 22 of them in an ILT gradient).  Kernels
// with tensor memory allocate it after the wait (a block holding tensor
// memory while it waits could keep the running kernel from allocating its
// own).
#pragma once
#include <cuda_runtime.h>

namespace huv_dev {
__device__ __forceinline__ void pdl_begin() {
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  asm volatile("griddepcontrol.wait;" ::: "memory");
}
}  // namespace huv_dev

namespace huv_launch {
// Grids of at most eight blocks per SM, outside graph capture: a launch hides
// behind the kernel before it (one 256^2 clip 31.5 -> 25.9 us, an ILT gradient
// of three 159 -> 131 us), but waiting blocks beside a long grid's tail cost
// more than its launch (64 masks of 1024^2 1.420 -> 1.430 ms with every launch
// programmatic), and so do they beside the other branches of a captured plan
// (90 clips 0.194 -> 0.231 ms).
constexpr unsigned kPdlBlocks = 8 * 148;
inline bool pdl_ok(dim3 grid, cudaStream_t st) {
  if (static_cast<unsigned long long>(grid.x) * grid.y * grid.z > kPdlBlocks) return false;
  cudaStreamCaptureStatus c = cudaStreamCaptureStatusNone;
  return st == nullptr || (cudaStreamIsCapturing(st, &c) == cudaSuccess && c == cudaStreamCaptureStatusNone);
}

template <typename... P, typename... A>
cudaError_t pdl(void (*kernel)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t st, A... args) {
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = at;
  cfg.numAttrs = pdl_ok(grid, st) ? 1 : 0;
  return cudaLaunchKernelEx(&cfg, kernel, static_cast<P>(args)...);
}
}  // namespace huv_launch
