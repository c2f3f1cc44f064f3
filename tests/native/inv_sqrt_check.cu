// Compares inv_sqrt (and the range-limited forms under it) with IEEE
// 1 / sqrt(x) for every binary32 bit pattern, on the device.  Prints the
// number of differing patterns: total, and of sqrt_from_estimate and
// inv_sqrt_in_range inside the range they are stated for.
#include <cstdio>

#include "rfmm_device.cuh"

using namespace rfmm;

__global__ void check(unsigned long long *bad) {
  const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
  for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < (1ull << 32); i += stride) {
    const float x = __uint_as_float((uint32_t)i);
    const float root = sqrtf(x), want = 1.0f / root, got = inv_sqrt(x);
    // NaN payloads are not part of the contract.
    if (want != want ? got == got : __float_as_uint(got) != __float_as_uint(want)) atomicAdd(bad, 1ull);
    if (x >= 0x1p-100f && x < 0x1p127f) {
      if (__float_as_uint(sqrt_from_estimate(x, rsqrt_estimate(x))) != __float_as_uint(root)) atomicAdd(bad + 1, 1ull);
      if (__float_as_uint(inv_sqrt_in_range(x)) != __float_as_uint(want)) atomicAdd(bad + 2, 1ull);
    }
  }
}

int main() {
  unsigned long long *d = nullptr, h[3] = {1, 1, 1};
  if (cudaMalloc(&d, sizeof(h)) != cudaSuccess || cudaMemset(d, 0, sizeof(h)) != cudaSuccess) return 2;
  check<<<1216, 256>>>(d);
  if (cudaMemcpy(h, d, sizeof(h), cudaMemcpyDeviceToHost) != cudaSuccess) return 2;
  std::printf("%llu %llu %llu\n", h[0], h[1], h[2]);
  return h[0] + h[1] + h[2] == 0 ? 0 : 1;
}
