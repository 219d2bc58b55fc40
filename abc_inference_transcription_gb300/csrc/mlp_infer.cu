// mlp_infer.cu — the surrogate ensemble's passes over all layers in one kernel
// on the tcgen05 tensor cores: the forward pass for prediction, and for training the
// forward pass that keeps what the backward pass reads, and the chain of derivatives.
//
// A CTA takes a tile of 128 rows of one member through the network: the
// activations stay in shared memory (BF16, 64 KB, K-major with the 128-byte
// swizzle the MMA reads), the accumulators in 256 columns of tensor memory,
// and only the input rows (32 B each) are read and the outputs written.  Layer
// by layer through global memory (mlp_forward), every hidden layer's BF16
// activations were written and read again and each tile was its own CTA with
// no overlap.  500,000 rows x 4 members: 1.4 ms against 4.7.
//
// Roles: warp 16 streams the weights (64 x 128 BF16 boxes, 16 KB, from L2: all
// members' weights are 1.3 MB) through a 3-stage ring and loads the tile's
// input rows; one lane of warp 17 issues the MMAs (M = N = 128, K = 16; the same
// shapes and order over K as mlp_tc.cu, so the results are bit-identical);
// warps 0-15 (four per TMEM lane quarter, 64 columns each) add the bias, apply
// SiLU and write the next layer's operand in place, once all MMAs of the layer
// have read the old one.  113 KB of shared memory and 256 TMEM columns per CTA
// let two CTAs share an SM, so that one's epilogue (0.09 ms of MUFU work per 4 x
// 65,536 rows, 0.18 ms with its other instructions) runs beside the other's
// MMAs and weight loads (0.11 ms on their own).  Waits are bounded as in mlp_tc.cu.
//
// Training (kFwd, kBwd): the same roles.  The forward pass also writes every
// hidden layer's pre-activations and transposed activations; the backward chain
// starts from dY and applies the layers' weights and the SiLU derivatives,
// writing the transposed dZ of each layer for the weight gradients.  Their
// global accesses go through shared memory in whole rows (mlp_tc.cuh), which leaves one CTA
// per SM.  4,096 rows x 4 members: 51 us in four launches of mlp_tc.cu and 39
// here forward, 40 in three and 32 here backward.
#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <atomic>
#include <cstring>

#include "kernels.h"
#include "mlp.cuh"
#include "mlp_tc.cuh"
#include "smem_attr.h"
#include "tcgen05.cuh"

namespace abc {
namespace {

using namespace tc;

constexpr int kRing = 3;
constexpr int kActChunks = kMlpHidden / kTcBK;     // 64-column chunks of the activations
constexpr uint32_t kChunkBytes = 128 * kTcBK * 2;  // 128 rows (or weight rows) x 64 values
constexpr int kInferSmem = (kActChunks + kRing) * (int)kChunkBytes + 128;
constexpr int kEpiWarps = 16, kEpiCols = kMlpHidden / (kEpiWarps / 4), kInferThreads = 32 * (kEpiWarps + 2);
constexpr uint32_t kInferTmem = 256;
enum PassKind { kPredict, kFwd, kBwd };
// the epilogue warps' staged chunks of the training passes
constexpr int kStageBytes = kEpiWarps * kChunk * kRowF * 4;
constexpr int pass_smem(PassKind kind) { return kInferSmem + (kind == kPredict ? 0 : kStageBytes); }
static_assert(pass_smem(kFwd) <= 227 * 1024, "one CTA's shared memory");

struct InferArgs {
  int B, nM, members, out_pad;
  int64_t b_off[4];
  int64_t n_params;
  const float* P;  // FP32 parameters (biases)
  float* Y;        // [members][B][out_pad]
  int* err;
  // training
  float* Z;             // [members][3][B][H] pre-activations (written by kFwd, read by kBwd)
  __nv_bfloat16* outT;  // kFwd: activations [members][3][H][ldT]; kBwd: dZ [layer][members][H][ldT]
  int ldT;
};

struct InferMaps {
  CUtensorMap x, w[4];
};

// Rows m_w .. m_w + 31 of member e, columns from kEpiCols part, of layer l of a
// training pass (kBwd counts from the last hidden layer down).
template <PassKind KIND>
__device__ __forceinline__ void train_epilogue(const InferArgs& g, uint8_t* smem, uint32_t lane_addr, int e, int m_w,
                                               int l, int part, int q4, int warp, int lane) {
  constexpr int H = kMlpHidden;
  float* sm = reinterpret_cast<float*>(smem + kInferSmem) + warp * kChunk * kRowF;
  const int rows = min(kChunk, g.B - m_w), row = q4 * 32 + lane;
  const int layer = KIND == kBwd ? 2 - l : l;
  const bool out = KIND == kFwd && l == 3, next = KIND == kFwd || l < 2;  // is there an operand to write
#pragma unroll 1
  for (int cc = 0; cc < kEpiCols / kChunk; ++cc) {
    const int col0 = part * kEpiCols + cc * kChunk;
    if (out && col0 >= g.out_pad) break;
    float x[kChunk];
    {
      uint32_t v[32];
      tmem_ld32(lane_addr + (uint32_t)col0, v);
#pragma unroll
      for (int j = 0; j < 32; ++j) x[j] = __uint_as_float(v[j]);
    }
    const int cols = out ? min(kChunk, g.out_pad - col0) : kChunk;
    float* z = g.Z + (((int64_t)e * 3 + layer) * g.B + m_w) * H + col0;
    if (KIND == kFwd) {
      const float* bias = g.P + e * g.n_params + g.b_off[l] + col0;
#pragma unroll
      for (int q = 0; q < 8; ++q) {
        if (4 * q >= cols) break;
        const float4 b = __ldg((const float4*)(bias + 4 * q));
        x[4 * q] += b.x; x[4 * q + 1] += b.y; x[4 * q + 2] += b.z; x[4 * q + 3] += b.w;
      }
      if (out) {
        store_rows_f32(sm, x, g.Y + ((int64_t)e * g.B + m_w) * g.out_pad + col0, g.out_pad, rows, cols, lane);
        continue;
      }
      store_rows_f32(sm, x, z, H, rows, kChunk, lane);
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        float xq[8], sg[8];
#pragma unroll
        for (int j = 0; j < 8; ++j) xq[j] = x[8 * q + j];
        sigm8(xq, sg);
#pragma unroll
        for (int j = 0; j < 8; ++j) x[8 * q + j] = xq[j] * sg[j];
      }
    } else {
      float zp[kChunk];
      load_rows_f32(sm, zp, z, H, rows, kChunk, lane);
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        float zq[8], sg[8];
#pragma unroll
        for (int j = 0; j < 8; ++j) zq[j] = zp[8 * q + j];
        sigm8(zq, sg);
#pragma unroll
        for (int j = 0; j < 8; ++j) x[8 * q + j] = x[8 * q + j] * (sg[j] * (1.0f + zq[j] * (1.0f - sg[j])));
      }
    }
    __nv_bfloat16* oT = KIND == kFwd ? g.outT + ((int64_t)e * 3 + layer) * H * g.ldT
                                     : g.outT + ((int64_t)layer * g.members + e) * H * g.ldT;
    oT += (int64_t)col0 * g.ldT + m_w + lane;
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      __nv_bfloat16 h[8];
#pragma unroll
      for (int j = 0; j < 8; ++j) h[j] = __float2bfloat16(x[8 * q + j]);
      if (lane < rows) {
#pragma unroll
        for (int j = 0; j < 8; ++j) oT[(int64_t)(8 * q + j) * g.ldT] = h[j];
      }
      if (next) {  // the next layer's operand, as in the prediction
        uint4 pk;
        memcpy(&pk, h, 16);
        const int col = col0 + 8 * q, unit = (col >> 3) & 7;
        *(uint4*)(smem + (col >> 6) * kChunkBytes + row * 128 + ((unit ^ (row & 7)) << 4)) = pk;
      }
    }
  }
}

template <PassKind KIND>
__global__ void __launch_bounds__(kInferThreads, KIND == kPredict ? 2 : 1)
    mlp_infer_kernel(const __grid_constant__ InferMaps maps, InferArgs g) {
  extern __shared__ __align__(1024) uint8_t smem[];
  uint8_t* ring = smem + kActChunks * kChunkBytes;
  uint64_t* full = (uint64_t*)(ring + kRing * kChunkBytes);
  uint64_t* empty = full + kRing;
  uint64_t* xfull = empty + kRing;
  uint64_t* acc_full = xfull + 1;
  uint64_t* act_ready = acc_full + 1;
  uint64_t* act_free = act_ready + 1;  // once per tile, where acc_full completes once per layer
  uint64_t* drain = act_free + 1;
  uint32_t* tslot = (uint32_t*)(drain + 1);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t sbase = su32(smem);
  if (sbase & 1023u) {  // the swizzle needs it; the same for every thread
    if (threadIdx.x == 0) atomicOr(g.err, 16);
    return;
  }
  if (threadIdx.x == 0) {
    for (int i = 0; i < kRing; ++i) {
      mbar_init(&full[i], 1);
      mbar_init(&empty[i], 1);
    }
    mbar_init(xfull, 1);
    mbar_init(acc_full, 1);
    mbar_init(act_ready, 32 * kEpiWarps);
    mbar_init(act_free, 1);
    mbar_init(drain, 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(su32(tslot)),
                 "r"(kInferTmem)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tbase = *tslot;
  const int tiles = g.nM * g.members;
  // layers of the pass; K chunks and N halves of each
  constexpr int L = KIND == kBwd ? 3 : 4;
  const int out_tiles = (g.out_pad + 127) / 128;  // 1 or 2
  const int in_chunks = KIND == kBwd ? (g.out_pad + kTcBK - 1) / kTcBK : 1;
  auto chunks_of = [&](int l) { return l == 0 ? in_chunks : kActChunks; };
  auto halves_of = [&](int l) { return KIND != kBwd && l == 3 ? out_tiles : 2; };

  if (warp == kEpiWarps) {
    if (lane == 0) {
      // ---- TMA producer
      int last_par[kRing] = {-1, -1, -1};
      int st = 0, ti = 0, x_par = -1;
      uint32_t ph = 0;
      bool ok = true;
      for (int t = blockIdx.x; t < tiles && ok; t += gridDim.x, ++ti) {
        const int e = t / g.nM, m0 = (t - e * g.nM) * 128;
        for (int l = 0; l < L && ok; ++l) {
          if (l == 0) {
            // the last layer of the previous tile has read the activations
            if (ti > 0 && !mbar_wait(act_free, (uint32_t)(ti - 1) & 1u)) {
              ok = false;
              break;
            }
            mbar_expect_tx(xfull, in_chunks * kChunkBytes);
            for (int c = 0; c < in_chunks; ++c)
              tma_load3(sbase + c * kChunkBytes, &maps.x, xfull, c * kTcBK, m0, KIND == kPredict ? 0 : e);
            x_par = ti & 1;
          }
          const int chunks = chunks_of(l), halves = halves_of(l);
          for (int c = 0; c < chunks && ok; ++c)
            for (int h = 0; h < halves; ++h) {
              if (!mbar_wait(&empty[st], ph ^ 1u)) {
                ok = false;
                break;
              }
              mbar_expect_tx(&full[st], kChunkBytes);
              tma_load3(su32(ring) + st * kChunkBytes, &maps.w[l], &full[st], c * kTcBK, h * 128, e);
              last_par[st] = (int)ph;
              if (++st == kRing) {
                st = 0;
                ph ^= 1u;
              }
            }
        }
      }
      if (!ok) atomicOr(g.err, 1);
      // copies in flight land before the CTA leaves
      for (int i = 0; i < kRing; ++i)
        if (last_par[i] >= 0 && !mbar_wait(&full[i], (uint32_t)last_par[i])) atomicOr(g.err, 8);
      if (x_par >= 0 && !mbar_wait(xfull, (uint32_t)x_par)) atomicOr(g.err, 8);
    }
  } else if (warp == kEpiWarps + 1) {
    if (lane == 0) {
      // ---- MMA issuer; n counts layers over all tiles
      int st = 0, n = 0, ti = 0;
      uint32_t ph = 0;
      bool ok = true;
      for (int t = blockIdx.x; t < tiles && ok; t += gridDim.x, ++ti) {
        for (int l = 0; l < L && ok; ++l, ++n) {
          // the epilogue of the layer before has written the operand and read the accumulators
          if (n > 0 && !mbar_wait(act_ready, (uint32_t)(n - 1) & 1u)) ok = false;
          if (ok && l == 0 && !mbar_wait(xfull, (uint32_t)ti & 1u)) ok = false;
          if (!ok) break;
          const int chunks = chunks_of(l), halves = halves_of(l);
          for (int c = 0; c < chunks && ok; ++c)
            for (int h = 0; h < halves; ++h) {
              if (!mbar_wait(&full[st], ph)) {
                ok = false;
                break;
              }
              tc_fence_after();
              const uint64_t da = sw128_desc(sbase + c * kChunkBytes);
              const uint64_t db = sw128_desc(su32(ring) + st * kChunkBytes);
#pragma unroll
              for (int kk = 0; kk < kTcBK / 16; ++kk)
                mma_bf16_128(tbase + (uint32_t)(h * 128), da + (uint64_t)(kk * 2), db + (uint64_t)(kk * 2),
                             (c > 0 || kk > 0) ? 1u : 0u);
              mma_commit(&empty[st]);
              if (++st == kRing) {
                st = 0;
                ph ^= 1u;
              }
            }
          if (ok) mma_commit(acc_full);
          if (ok && l == L - 1) mma_commit(act_free);
        }
      }
      if (!ok) atomicOr(g.err, 2);
      mma_commit(drain);  // every MMA issued has finished before the tensor memory is given back
      if (!mbar_wait(drain, 0)) atomicOr(g.err, 32);
    }
  } else {
    // ---- epilogue: TMEM lane quarter = warp % 4, columns from kEpiCols (warp / 4)
    const int q = warp & 3, part = warp >> 2;
    const int row = q * 32 + lane;
    const uint32_t lane_addr = tbase + ((uint32_t)(q * 32) << 16);
    int n = 0;
    bool ok = true;
    for (int t = blockIdx.x; t < tiles && ok; t += gridDim.x) {
      const int e = t / g.nM;
      const int64_t m = (int64_t)(t - e * g.nM) * 128 + row;
      for (int l = 0; l < L; ++l, ++n) {
        ok = __all_sync(0xffffffffu, mbar_wait(acc_full, (uint32_t)n & 1u));
        if (!ok) {
          if (lane == 0) atomicOr(g.err, 4);
          break;
        }
        tc_fence_after();
        if (KIND != kPredict) {
          train_epilogue<KIND>(g, smem, lane_addr, e, (t - e * g.nM) * 128 + q * 32, l, part, q, warp, lane);
          asm volatile("fence.proxy.async.shared::cta;" ::: "memory");  // the MMAs read what was just written
          tc_fence_before();
          mbar_arrive(act_ready);
          continue;
        }
        const float* bias = g.P + e * g.n_params + g.b_off[l];
#pragma unroll 1
        for (int cc = 0; cc < kEpiCols / 16; ++cc) {
          const int col0 = part * kEpiCols + cc * 16;
          if (l == 3 && col0 >= g.out_pad) break;
          uint32_t v[16];
          tmem_ld16(lane_addr + (uint32_t)col0, v);
#pragma unroll
          for (int j = 0; j < 2; ++j) {
            const int col = col0 + 8 * j;
            const float4 b0 = __ldg((const float4*)(bias + col)), b1 = __ldg((const float4*)(bias + col + 4));
            const float x[8] = {__uint_as_float(v[8 * j]) + b0.x,     __uint_as_float(v[8 * j + 1]) + b0.y,
                          __uint_as_float(v[8 * j + 2]) + b0.z, __uint_as_float(v[8 * j + 3]) + b0.w,
                          __uint_as_float(v[8 * j + 4]) + b1.x, __uint_as_float(v[8 * j + 5]) + b1.y,
                          __uint_as_float(v[8 * j + 6]) + b1.z, __uint_as_float(v[8 * j + 7]) + b1.w};
            if (l < 3) {
              // 16 bytes of the swizzled row: unit (col / 8) % 8 exchanged with the row's low bits
              __nv_bfloat16 h[8];
              float sg[8];
              sigm8(x, sg);
#pragma unroll
              for (int i = 0; i < 8; ++i) h[i] = __float2bfloat16(x[i] * sg[i]);
              uint4 pk;
              memcpy(&pk, h, 16);
              const int unit = (col >> 3) & 7;
              *(uint4*)(smem + (col >> 6) * kChunkBytes + row * 128 + ((unit ^ (row & 7)) << 4)) = pk;
            } else if (m < g.B) {
              float* o = g.Y + ((int64_t)e * g.B + m) * g.out_pad + col;
              *(float4*)o = make_float4(x[0], x[1], x[2], x[3]);
              *(float4*)(o + 4) = make_float4(x[4], x[5], x[6], x[7]);
            }
          }
        }
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");  // the MMAs read what was just written
        tc_fence_before();
        mbar_arrive(act_ready);
      }
    }
  }
  __syncwarp();
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  if (warp == 0)
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tbase), "r"(kInferTmem));
}

}  // namespace

bool mlp_infer_fits(const MlpDims& d) { return d.H == kMlpHidden && d.in_pad <= kTcBK && d.out_pad <= 256; }

template <PassKind KIND>
static cudaError_t launch_pass(const InferMaps& maps, const InferArgs& g, int sms, cudaStream_t s) {
  static std::atomic<uint64_t> attr{0};
  cudaError_t e = set_smem_once(attr, mlp_infer_kernel<KIND>, pass_smem(KIND));
  if (e != cudaSuccess) return e;
  const int grid = (int)std::min<int64_t>((int64_t)g.nM * g.members, (KIND == kPredict ? 2 : 1) * (int64_t)sms);
  mlp_infer_kernel<KIND><<<grid, kInferThreads, pass_smem(KIND), s>>>(maps, g);
  return cudaGetLastError();
}

static InferArgs pass_args(const MlpDims& d, int members, int B, const float* Pf, float* Y, int* err) {
  InferArgs g{};
  const int64_t b_off[4] = {d.off_b1, d.off_b2, d.off_b3, d.off_b4};
  for (int l = 0; l < 4; ++l) g.b_off[l] = b_off[l];
  g.B = B;
  g.nM = (B + 127) / 128;
  g.members = members;
  g.out_pad = d.out_pad;
  g.n_params = d.n_params;
  g.P = Pf;
  g.Y = Y;
  g.err = err;
  return g;
}

// weights of the forward passes: W^T [N][K] of every layer
static bool forward_maps(const MlpDims& d, int members, const __nv_bfloat16* WhT, InferMaps* maps) {
  const int64_t w_off[4] = {d.off_w1, d.off_w2, d.off_w3, d.off_w4};
  for (int l = 0; l < 4; ++l) {
    const int K = l == 0 ? d.in_pad : d.H, N = l == 3 ? d.out_pad : d.H;
    if (!make_map3(&maps->w[l], WhT + w_off[l], K, K, N, members, d.n_params)) return false;
  }
  return true;
}

cudaError_t mlp_infer(const MlpDims& d, int members, int B, const __nv_bfloat16* X0, const __nv_bfloat16* WhT,
                      const float* Pf, float* Y, int* err, int sms, cudaStream_t s) {
  if (B <= 0) return cudaSuccess;
  InferMaps maps;
  if (!make_map3(&maps.x, X0, d.in_pad, d.in_pad, B, 1, 0) || !forward_maps(d, members, WhT, &maps))
    return cudaErrorInvalidValue;
  return launch_pass<kPredict>(maps, pass_args(d, members, B, Pf, Y, err), sms, s);
}

// X0: [members][B][in_pad]
cudaError_t mlp_train_forward(const MlpDims& d, int members, int B, const __nv_bfloat16* X0, const __nv_bfloat16* WhT,
                              const float* Pf, float* Z, __nv_bfloat16* AhT, int ldT, float* Y, int* err, int sms,
                              cudaStream_t s) {
  if (B <= 0) return cudaSuccess;
  InferMaps maps;
  if (!make_map3(&maps.x, X0, d.in_pad, d.in_pad, B, members, (int64_t)B * d.in_pad) ||
      !forward_maps(d, members, WhT, &maps))
    return cudaErrorInvalidValue;
  InferArgs g = pass_args(d, members, B, Pf, Y, err);
  g.Z = Z;
  g.outT = AhT;
  g.ldT = ldT;
  return launch_pass<kFwd>(maps, g, sms, s);
}

// dY: [members][B][out_pad]; Wh: the weights as stored, W_l [H][out], K-major for dZ_{l-1} = dZ_l W_l^T
cudaError_t mlp_train_backward(const MlpDims& d, int members, int B, const __nv_bfloat16* dY, const __nv_bfloat16* Wh,
                               float* Z, __nv_bfloat16* dZT, int ldT, int* err, int sms, cudaStream_t s) {
  if (B <= 0) return cudaSuccess;
  InferMaps maps;
  const int64_t w_off[3] = {d.off_w4, d.off_w3, d.off_w2};
  if (!make_map3(&maps.x, dY, d.out_pad, d.out_pad, B, members, (int64_t)B * d.out_pad)) return cudaErrorInvalidValue;
  for (int l = 0; l < 3; ++l) {
    const int K = l == 0 ? d.out_pad : d.H;
    if (!make_map3(&maps.w[l], Wh + w_off[l], K, K, d.H, members, d.n_params)) return cudaErrorInvalidValue;
  }
  maps.w[3] = maps.w[2];
  InferArgs g = pass_args(d, members, B, nullptr, nullptr, err);
  g.Z = Z;
  g.outT = dZT;
  g.ldT = ldT;
  return launch_pass<kBwd>(maps, g, sms, s);
}

}  // namespace abc
