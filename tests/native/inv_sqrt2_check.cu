// The packed forms of inv_sqrt_check.cu's functions, on the device: every
// binary32 pattern in the low half, another one in the high half (i -> a i + c
// runs through every pattern too, so halves inside and outside the range of
// the division-free path meet).  Prints the number of patterns for which
// inv_sqrt2, sqrt2<false>, sqrt2<true> (2^-100 and above) and
// inv_sqrt2_in_range (both halves in its range) differ from IEEE operations.
#include <cstdio>

#include "rfmm_device.cuh"

using namespace rfmm;

__device__ bool differs(float got, float want) {
  return want != want ? got == got : __float_as_uint(got) != __float_as_uint(want);  // any NaN will do
}

__global__ void check(unsigned long long *bad, float minus_zero) {
  const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
  const f32x2 mz = pack2(minus_zero, minus_zero);
  for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < (1ull << 32); i += stride) {
    const float x[2] = {__uint_as_float((uint32_t)i), __uint_as_float((uint32_t)i * 2654435761u + 97u)};
    const f32x2 v = pack2(x[0], x[1]);
    float inv[2], root[2], large[2], in_range[2];
    unpack2(inv_sqrt2(v, mz), inv[0], inv[1]);
    unpack2(sqrt2<false>(v, mz), root[0], root[1]);
    const float lo[2] = {x[0] >= 0x1p-100f ? x[0] : 1.0f, x[1] >= 0x1p-100f ? x[1] : 1.0f};
    unpack2(sqrt2<true>(pack2(lo[0], lo[1]), mz), large[0], large[1]);
    const float in[2] = {lo[0] < 0x1p127f ? lo[0] : 2.0f, lo[1] < 0x1p127f ? lo[1] : 2.0f};
    unpack2(inv_sqrt2_in_range(pack2(in[0], in[1]), in[0], in[1], mz), in_range[0], in_range[1]);
    for (int h = 0; h < 2; h++) {
      if (differs(inv[h], 1.0f / sqrtf(x[h]))) atomicAdd(bad, 1ull);
      if (differs(root[h], sqrtf(x[h]))) atomicAdd(bad + 1, 1ull);
      if (differs(large[h], sqrtf(lo[h]))) atomicAdd(bad + 2, 1ull);
      if (differs(in_range[h], 1.0f / sqrtf(in[h]))) atomicAdd(bad + 3, 1ull);
    }
  }
}

int main() {
  unsigned long long *d = nullptr, h[4] = {1, 1, 1, 1};
  if (cudaMalloc(&d, sizeof(h)) != cudaSuccess || cudaMemset(d, 0, sizeof(h)) != cudaSuccess) return 2;
  check<<<1216, 256>>>(d, -0.0f);
  if (cudaMemcpy(h, d, sizeof(h), cudaMemcpyDeviceToHost) != cudaSuccess) return 2;
  std::printf("%llu %llu %llu %llu\n", h[0], h[1], h[2], h[3]);
  return h[0] + h[1] + h[2] + h[3] == 0 ? 0 : 1;
}
