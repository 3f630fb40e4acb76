// sqrt_ge1 (the root of every ns-mode weight) against __fsqrt_rn over all floats from 1 to infinity.  Built by
// tests/test_gpu_sqrt.py.
#include <cstdint>
#include <cuda_runtime.h>

#include "dtb_device.cuh"

__global__ void sweep(uint32_t first, uint32_t last, unsigned long long* out) {
  unsigned long long bad = 0;
  for (uint64_t b = first + (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; b <= last; b += (uint64_t)gridDim.x * blockDim.x) {
    const float x = __uint_as_float((uint32_t)b);
    if (__float_as_uint(dtb::sqrt_ge1(x)) != __float_as_uint(__fsqrt_rn(x))) {
      ++bad;
      atomicMin(&out[1], (unsigned long long)b);
    }
  }
  if (bad) atomicAdd(&out[0], bad);
}

// out: the number of floats (bit patterns first .. last) whose roots differ, and the smallest of them.
extern "C" __attribute__((visibility("default"))) int sqrt_mismatches(uint32_t first, uint32_t last, unsigned long long* out) {
  unsigned long long* dev = nullptr;
  out[0] = 0;
  out[1] = ~0ull;
  if (cudaMalloc(&dev, 16) != cudaSuccess) return -1;
  bool ok = cudaMemcpy(dev, out, 16, cudaMemcpyHostToDevice) == cudaSuccess;
  sweep<<<148 * 8, 256>>>(first, last, dev);
  ok = ok && cudaDeviceSynchronize() == cudaSuccess && cudaMemcpy(out, dev, 16, cudaMemcpyDeviceToHost) == cudaSuccess;
  cudaFree(dev);
  return ok ? 0 : -1;
}
