// mlp_tc.cuh — what the surrogate's tensor-core kernels (mlp_tc.cu,
// mlp_infer.cu) share: the BF16 MMA of a 128 x 128 tile, the sigmoid of the
// epilogues and the tensor maps of their operands.
#pragma once
#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>

namespace abc {
namespace tc {

constexpr int kTcBK = 64;  // BF16 values along K per box = one 128-byte swizzled row

// D = F32, A = B = BF16, both K-major, M = N = 128
constexpr uint32_t kIdescBf16 =
    (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(128 >> 3) << 17) | ((uint32_t)(128 >> 4) << 24);

__device__ __forceinline__ void mma_bf16_128(uint32_t d_tmem, uint64_t a, uint64_t b, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}" ::"r"(d_tmem),
      "l"(a), "l"(b), "r"(kIdescBf16), "r"(accumulate)
      : "memory");
}

// 1 / y for y in [1, 2^126): one Newton step on the hardware approximation
// (P. Markstein, IBM J. Res. Dev. 34(1), 1990).  Correctly rounded over that
// range, i.e. equal to the IEEE division, as checked over every float of it
// by tests/test_surrogate_kernels.py; no scaling and no slow path.
__device__ __forceinline__ float recip_ge1(float y) {
  float r;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(y));
  return fmaf(r, fmaf(-y, r, 1.0f), r);
}

// exp(-z) = 2^(-z log2 e) on the hardware approximation with subnormals as
// zero: 1 + exp(-z) equals that of __expf(-z) for every z > -87 (same test).
__device__ __forceinline__ float exp_neg(float z) {
  float e;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(e) : "f"(z * -1.4426950408889634f));
  return e;
}

// s[j] = 1 / (1 + exp(-z[j])): beyond z = -87 the denominator leaves the range
// of recip_ge1 and its quotient may be subnormal, so the division is used (its
// loop unrolled: indexed, the arrays would live in local memory).  The fused
// forward pass over 4 x 65,536 rows: 0.18 ms with this, 0.34 with the division
// alone, whose slow path interrupts every activation.
__device__ __forceinline__ void sigm8(const float (&z)[8], float (&s)[8]) {
  float lo = z[0];
#pragma unroll
  for (int j = 1; j < 8; ++j) lo = fminf(lo, z[j]);
#pragma unroll
  for (int j = 0; j < 8; ++j) s[j] = recip_ge1(1.0f + exp_neg(z[j]));
  if (lo <= -87.0f) {
#pragma unroll
    for (int j = 0; j < 8; ++j) s[j] = 1.0f / (1.0f + __expf(-z[j]));
  }
}

constexpr int kChunk = 32;  // rows and columns of an epilogue chunk
// row strides of a staged chunk, in words: 16-byte pieces of eight neighbouring lanes fall
// on distinct banks, by rows and by columns
constexpr int kRowF = kChunk + 4, kRowH = kChunk / 2 + 4;

// What bounds the epilogue is the load/store path: a lane holds a row of the chunk, and a
// 16-byte access per lane touches 32 rows.  Through shared memory the warp's
// accesses take whole rows instead, 4 (FP32) or 8 (BF16) of them at a time.
// rows, cols: what of the chunk is inside the matrix.
__device__ __forceinline__ void store_rows_f32(float* sm, const float (&x)[kChunk], float* base, int64_t ld, int rows,
                                               int cols, int lane) {
#pragma unroll
  for (int q = 0; q < 8; ++q)
    *(float4*)(sm + lane * kRowF + 4 * q) = make_float4(x[4 * q], x[4 * q + 1], x[4 * q + 2], x[4 * q + 3]);
  __syncwarp();
  const int r = lane / 8, c = lane % 8 * 4;
#pragma unroll
  for (int t = 0; t < 8; ++t)
    if (4 * t + r < rows && c < cols) *(float4*)(base + (4 * t + r) * ld + c) = *(const float4*)(sm + (4 * t + r) * kRowF + c);
  __syncwarp();
}

__device__ __forceinline__ void load_rows_f32(float* sm, float (&x)[kChunk], const float* base, int64_t ld, int rows,
                                              int cols, int lane) {
  const int r = lane / 8, c = lane % 8 * 4;
  float4 v[8];
#pragma unroll
  for (int t = 0; t < 8; ++t)
    v[t] = 4 * t + r < rows && c < cols ? *(const float4*)(base + (4 * t + r) * ld + c) : make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
  for (int t = 0; t < 8; ++t) *(float4*)(sm + (4 * t + r) * kRowF + c) = v[t];
  __syncwarp();
#pragma unroll
  for (int q = 0; q < 8; ++q) {
    const float4 w = *(const float4*)(sm + lane * kRowF + 4 * q);
    x[4 * q] = w.x; x[4 * q + 1] = w.y; x[4 * q + 2] = w.z; x[4 * q + 3] = w.w;
  }
  __syncwarp();
}

// 3D map over [members][rows][K] BF16 (K contiguous): box 64 x 128 x 1, 128-byte swizzle
bool make_map3(CUtensorMap* map, const __nv_bfloat16* base, int64_t K, int64_t ld, int64_t rows, int64_t members,
               int64_t member_stride);

}  // namespace tc
}  // namespace abc
