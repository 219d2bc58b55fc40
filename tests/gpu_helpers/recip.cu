// abc::tc::recip_ge1 against the IEEE division, for every float in [1, 2^126),
// and sigm8 against 1 / (1 + __expf(-z)) for every float z.
#include <cuda_runtime.h>

#include <cstdint>

#include "../../abc_inference_transcription_gb300/csrc/mlp_tc.cuh"

__global__ void recip_kernel(uint32_t first, uint32_t last, unsigned long long* bad) {
  for (uint64_t b = first + blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; b < last;
       b += (uint64_t)gridDim.x * blockDim.x) {
    const float y = __uint_as_float((uint32_t)b);
    if (__float_as_uint(abc::tc::recip_ge1(y)) != __float_as_uint(1.0f / y)) atomicAdd(bad, 1ull);
  }
}

__global__ void sigm_kernel(unsigned long long* bad) {
  for (uint64_t b = 8 * (blockIdx.x * (uint64_t)blockDim.x + threadIdx.x); b < (1ull << 32);
       b += 8 * (uint64_t)gridDim.x * blockDim.x) {
    float z[8], s[8];
    for (int j = 0; j < 8; ++j) z[j] = __uint_as_float((uint32_t)(b + j));
    abc::tc::sigm8(z, s);
    for (int j = 0; j < 8; ++j) {
      const float want = 1.0f / (1.0f + __expf(-z[j]));
      if (__float_as_uint(s[j]) != __float_as_uint(want) && !(s[j] != s[j] && want != want)) atomicAdd(bad, 1ull);
    }
  }
}

extern "C" int recip_check(unsigned long long* bad_out) {
  unsigned long long* d = nullptr;
  if (cudaMalloc(&d, 2 * sizeof(*d)) != cudaSuccess) return 1;
  cudaMemset(d, 0, 2 * sizeof(*d));
  recip_kernel<<<4096, 256>>>(0x3f800000u, 0x7e800000u, d);  // 1 and 2^126
  sigm_kernel<<<4096, 256>>>(d + 1);
  cudaError_t e = cudaDeviceSynchronize();
  if (e == cudaSuccess) e = cudaMemcpy(bad_out, d, 2 * sizeof(*d), cudaMemcpyDeviceToHost);
  cudaFree(d);
  return e == cudaSuccess ? 0 : 1;
}
