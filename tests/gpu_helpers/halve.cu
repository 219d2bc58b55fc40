// The production SSA's two forms of Bin(n, 1/2) at division -- one lane alone
// (lane_halve) and the whole warp (warp_halve) -- for n = 0 .. count - 1.
#include <cuda_runtime.h>

#include "../../abc_inference_transcription_gb300/csrc/ssa_fp32.cuh"

struct Keys {
  uint32_t rk[20];
};

__global__ void halve_kernel(Keys keys, int count, int* out) {
  const int n = blockIdx.x, lane = threadIdx.x;
  uint32_t b1 = 3u << 24, b2 = 3u << 24;
  const int w = abc::warp_halve(n, b1, 17u, 23u, lane, keys.rk);
  const int l = abc::lane_halve(n, b2, 17u, 23u, keys.rk);
  if (lane == 0) {
    out[4 * n] = w;
    out[4 * n + 1] = l;
    out[4 * n + 2] = (int)b1;
    out[4 * n + 3] = (int)b2;
  }
}

// out: 4 x count: both counts, and the block counter after each
extern "C" int halve_counts(unsigned long long seed, int count, int* out) {
  Keys k;
  uint32_t k0 = (uint32_t)seed, k1 = (uint32_t)(seed >> 32);
  for (int r = 0; r < 10; ++r) {
    k.rk[2 * r] = k0;
    k.rk[2 * r + 1] = k1;
    k0 += 0x9E3779B9u;
    k1 += 0xBB67AE85u;
  }
  int* d = nullptr;
  if (cudaMalloc(&d, sizeof(int) * 4 * (size_t)count) != cudaSuccess) return 1;
  halve_kernel<<<count, 32>>>(k, count, d);
  cudaError_t e = cudaDeviceSynchronize();
  if (e == cudaSuccess) e = cudaMemcpy(out, d, sizeof(int) * 4 * (size_t)count, cudaMemcpyDeviceToHost);
  cudaFree(d);
  return e == cudaSuccess ? 0 : 1;
}
