// gelu_bf16x2 (csrc/cuda/fno_gelu.cuh) against the BF16 rounding of gelu_erf
// for every FP32 bit pattern, each in both places of a pair.  Prints the
// number of patterns whose bits differ.
#include <cstdio>

#include "../highuvlith_b200/csrc/cuda/fno_gelu.cuh"
using namespace huv_dev;

__global__ void check(unsigned long long* bad) {
  unsigned long long n = 0;
  for (unsigned long long i = blockIdx.x * 256ull + threadIdx.x; i < (1ull << 32); i += gridDim.x * 256ull) {
    const float x = __uint_as_float(static_cast<unsigned>(i)), y = __uint_as_float(static_cast<unsigned>(i) ^ 0x5a5a5au);
    const __nv_bfloat162 g = gelu_bf16x2(x, y), r = __floats2bfloat162_rn(gelu_erf(x), gelu_erf(y));
    n += *reinterpret_cast<const unsigned*>(&g) != *reinterpret_cast<const unsigned*>(&r);
  }
  if (n) atomicAdd(bad, n);
}

int main() {
  unsigned long long *d, h = 0;
  if (cudaMalloc(&d, 8) != cudaSuccess || cudaMemset(d, 0, 8) != cudaSuccess) return 2;
  check<<<148 * 8, 256>>>(d);
  if (cudaMemcpy(&h, d, 8, cudaMemcpyDeviceToHost) != cudaSuccess) return 2;
  printf("%llu\n", h);
  return 0;
}
