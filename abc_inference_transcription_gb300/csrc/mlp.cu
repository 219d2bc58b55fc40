// mlp.cu — forward, backward and Adam of the surrogate ensemble.  Every GEMM
// runs on the tcgen05 tensor cores (mlp_tc.cu) with both operands K-major, so
// the passes keep transposed BF16 copies where the backward pass reduces over
// the batch: W^T for the forward GEMMs, and X0^T, A_l^T, dY^T, dZ_l^T
// ([features][batch]) for the weight gradients.  See mlp.cuh for the layout.
#include <cuda_bf16.h>

#include <algorithm>

#include "common.cuh"
#include "kernels.h"
#include "mlp.cuh"
#include "sinhcosh.cuh"

namespace abc {

// ---------------------------------------------------------------------------
// elementwise kernels
// ---------------------------------------------------------------------------
// Glorot-uniform weights, zero biases and zero padding; Philox stream ST_AUX,
// cell = parameter block, particle = member.
__global__ void mlp_init_kernel(MlpDims d, int members, uint64_t seed, float* P) {
  const int64_t n = d.n_params * members;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
    const int e = (int)(i / d.n_params);
    const int64_t q = i - (int64_t)e * d.n_params;
    float bound = 0.0f;
    bool valid = false;
    if (q >= d.off_w1 && q < d.off_b1) {
      const int64_t r = (q - d.off_w1) / d.H;
      valid = r < d.in_dim;
      bound = sqrtf(6.0f / (float)(d.in_dim + d.H));
    } else if ((q >= d.off_w2 && q < d.off_b2) || (q >= d.off_w3 && q < d.off_b3)) {
      valid = true;
      bound = sqrtf(6.0f / (float)(2 * d.H));
    } else if (q >= d.off_w4 && q < d.off_b4) {
      const int64_t c = (q - d.off_w4) % d.out_pad;
      valid = c < 2 * d.K;
      bound = 0.5f * sqrtf(6.0f / (float)(d.H + 2 * d.K));
    }
    float v = 0.0f;
    if (valid) {
      U4 c;
      c.x = (uint32_t)(q >> 2);
      c.y = (ST_AUX << 30) | 0x1000000u;
      c.z = (uint32_t)e;
      c.w = 0x4d4c5021u;
      U4 o = philox4x32_10(c, (uint32_t)seed, (uint32_t)(seed >> 32));
      const uint32_t w = (q & 3) == 0 ? o.x : (q & 3) == 1 ? o.y : (q & 3) == 2 ? o.z : o.w;
      v = bound * (2.0f * ((float)(w >> 8) * 5.9604644775390625e-08f) - 1.0f);
    }
    P[i] = v;
  }
}

__global__ void mlp_to_bf16_kernel(const float* src, __nv_bfloat16* dst, int64_t n) {
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
    dst[i] = __float2bfloat16(src[i]);
}

// BF16 transposed weights: W_l [R][C] at off_w -> W_l^T [C][R] at the same
// offset (biases copied), for the K-major forward GEMMs.
__global__ void mlp_weights_t_kernel(const float* P, MlpDims d, int members, __nv_bfloat16* PT) {
  const int64_t n = d.n_params * members;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
    const int64_t e = i / d.n_params, q = i - e * d.n_params;
    int64_t off = -1, R = 0, Cc = 0;
    if (q >= d.off_w1 && q < d.off_b1) { off = d.off_w1; R = d.in_pad; Cc = d.H; }
    else if (q >= d.off_w2 && q < d.off_b2) { off = d.off_w2; R = d.H; Cc = d.H; }
    else if (q >= d.off_w3 && q < d.off_b3) { off = d.off_w3; R = d.H; Cc = d.H; }
    else if (q >= d.off_w4 && q < d.off_b4) { off = d.off_w4; R = d.H; Cc = d.out_pad; }
    if (off < 0) {
      PT[i] = __float2bfloat16(P[i]);
    } else {
      const int64_t t = q - off, r = t / Cc, c = t - r * Cc;   // source element (r, c)
      PT[e * d.n_params + off + c * R + r] = __float2bfloat16(P[i]);
    }
  }
}

// rows of the batch for member e: idx = (a_e * (base + i) + b_e) mod N.  A
// block takes 32 rows: their indices once each (a 64-bit remainder), then the
// targets with a row's columns on neighbouring lanes and the inputs, whose
// transposed copy wants neighbouring rows, through shared memory.
constexpr int kGatherRows = 32;
__global__ void __launch_bounds__(256) mlp_gather_kernel(const float* xn, const float* yn, int64_t N, int in_pad, int K,
                                                         int B, int64_t base, const uint64_t* perm_ab,
                                                         __nv_bfloat16* X0, __nv_bfloat16* X0T, int ldT, float* T,
                                                         int64_t sX, int64_t sT) {
  __shared__ int64_t rows[kGatherRows];  // -1: past the end of the data
  __shared__ __nv_bfloat16 x[kGatherRows][kMlpInPad + 1];
  const int e = blockIdx.y, i0 = blockIdx.x * kGatherRows;
  const int nr = min(kGatherRows, B - i0);
  if ((int)threadIdx.x < nr) {
    const uint64_t a = perm_ab[2 * e], b = perm_ab[2 * e + 1];
    const int64_t pos = base + i0 + threadIdx.x;
    rows[threadIdx.x] = pos < N ? (int64_t)((a * (uint64_t)pos + b) % (uint64_t)N) : -1;
  }
  __syncthreads();
  for (int q = threadIdx.x; q < nr * in_pad; q += blockDim.x) {
    const int i = q / in_pad, c = q - i * in_pad;
    const int64_t r = rows[i];
    const __nv_bfloat16 v = __float2bfloat16(r >= 0 ? xn[r * in_pad + c] : 0.0f);
    X0[e * sX + (int64_t)i0 * in_pad + q] = v;
    x[i][c] = v;
  }
  for (int q = threadIdx.x; q < nr * K; q += blockDim.x) {
    const int i = q / K, k = q - i * K;
    const int64_t r = rows[i];
    T[e * sT + (int64_t)i0 * K + q] = r >= 0 ? yn[r * K + k] : __int_as_float(0x7fc00000);
  }
  if (!X0T) return;
  __syncthreads();
  for (int q = threadIdx.x; q < in_pad * kGatherRows; q += blockDim.x) {
    const int c = q / kGatherRows, i = q - c * kGatherRows;
    if (i < nr) X0T[(int64_t)e * in_pad * ldT + (int64_t)c * ldT + i0 + i] = x[i][c];
  }
}

// Gaussian negative log-likelihood on standardised targets; dY = dL/dY / count.
constexpr float kLvMin = -9.0f, kLvMax = 9.0f;

// A launch has two kinds of blocks.  The first sum the loss over the pairs in the
// order of nb blocks' grid-stride loops (a training run is reproducible bit for
// bit), kLossBlocks of them at a time: one each, the launch was four waves of blocks
// waiting for their loads (21 us for 4 x 4,096 rows of 53 statistics, 17 now).  The
// others take kLossRows rows of the gradient each, whose transposed copy goes
// through shared memory.
constexpr int kLossRows = 32, kLossBlocks = 4;
__global__ void __launch_bounds__(256) mlp_loss_kernel(const float* Y, const float* T, int B, int K, int out_pad,
                                                       float inv_count, __nv_bfloat16* dY, __nv_bfloat16* dYT, int ldT,
                                                       float* loss_part, int nb, int64_t sY, int64_t sT) {
  extern __shared__ __nv_bfloat16 tile[];  // [kLossRows][out_pad + 2]
  __shared__ float wsum[kLossBlocks][8];
  const int e = blockIdx.y, sum_blocks = (nb + kLossBlocks - 1) / kLossBlocks;
  if ((int)blockIdx.x < sum_blocks) {
    float local[kLossBlocks] = {};
    const int v0 = blockIdx.x * kLossBlocks, n = B * out_pad;
    for (int base = v0 * 256 + threadIdx.x; base < n; base += nb * 256) {
      float t[kLossBlocks], mu[kLossBlocks], lv_raw[kLossBlocks];
#pragma unroll
      for (int u = 0; u < kLossBlocks; ++u) {
        const int idx = base + u * 256;
        const int i = idx / out_pad, c = idx - (idx / out_pad) * out_pad;
        t[u] = __int_as_float(0x7fc00000);
        mu[u] = lv_raw[u] = 0.0f;
        if (v0 + u < nb && idx < n && c < K) {
          const float* y = Y + e * sY + idx;
          t[u] = T[e * sT + (int64_t)i * K + c];
          mu[u] = y[0];
          lv_raw[u] = y[K];
        }
      }
#pragma unroll
      for (int u = 0; u < kLossBlocks; ++u) {
        if (t[u] == t[u]) {
          const float lv = fminf(fmaxf(lv_raw[u], kLvMin), kLvMax);
          const float r = t[u] - mu[u];
          const float ei = __expf(-lv);
          local[u] += 0.5f * (lv + r * r * ei);
        }
      }
    }
    // block sums in a fixed order: warps by shuffles, then one thread over the warp sums
#pragma unroll
    for (int u = 0; u < kLossBlocks; ++u) {
      for (int o = 16; o > 0; o >>= 1) local[u] += __shfl_xor_sync(0xffffffffu, local[u], o);
      if ((threadIdx.x & 31) == 0) wsum[u][threadIdx.x >> 5] = local[u];
    }
    __syncthreads();
    if (threadIdx.x < kLossBlocks && v0 + (int)threadIdx.x < nb) {
      float t = 0.0f;
      for (int w = 0; w < 8; ++w) t += wsum[threadIdx.x][w];
      loss_part[e * nb + v0 + threadIdx.x] = t * inv_count;
    }
    return;
  }
  const int i0 = ((int)blockIdx.x - sum_blocks) * kLossRows, rows = min(kLossRows, B - i0), ld = out_pad + 2;
#pragma unroll 4
  for (int q = threadIdx.x; q < rows * K; q += blockDim.x) {
    const int i = q / K, k = q - i * K;
    const float* y = Y + e * sY + (int64_t)(i0 + i) * out_pad;
    const float t = T[e * sT + (int64_t)i0 * K + q], mu = y[k], lv_raw = y[K + k];
    float gm = 0.0f, gv = 0.0f;
    if (t == t) {
      const bool inside = lv_raw > kLvMin && lv_raw < kLvMax;
      const float lv = fminf(fmaxf(lv_raw, kLvMin), kLvMax);
      const float r = t - mu;
      const float ei = __expf(-lv);
      gm = -r * ei * inv_count;
      gv = inside ? 0.5f * (1.0f - r * r * ei) * inv_count : 0.0f;
    }
    tile[i * ld + k] = __float2bfloat16(gm);
    tile[i * ld + K + k] = __float2bfloat16(gv);
  }
  const int pad = out_pad - 2 * K;
  for (int q = threadIdx.x; q < rows * pad; q += blockDim.x)
    tile[q / pad * ld + 2 * K + q % pad] = __float2bfloat16(0.0f);
  __syncthreads();
  for (int q = threadIdx.x; q < rows * out_pad; q += blockDim.x) {
    const int i = q / out_pad, c = q - i * out_pad;
    dY[e * sY + (int64_t)i0 * out_pad + q] = tile[i * ld + c];
  }
  for (int q = threadIdx.x; q < out_pad * kLossRows; q += blockDim.x) {
    const int c = q / kLossRows, i = q - c * kLossRows;
    if (i < rows) dYT[(int64_t)e * out_pad * ldT + (int64_t)c * ldT + i0 + i] = tile[i * ld + c];
  }
}

// The reductions that end a backward pass, in one launch of three kinds of
// blocks (blockIdx.x), so that the two serial ones run beside the third:
//   columns  db[n] = sum_i dZ[i][n] for the output layer and the hidden ones, in
//            row order (a training run is reproducible bit for bit, and
//            independent of the launch), from the transposed copies [n][ldT].
//            The additions are one chain per column.  A warp takes kColsPerWarp
//            columns: it loads 256 rows of each at once (coalesced, the next 256 in
//            flight) and passes them through shared memory to the chains, four
//            lanes on one.  (A column per warp: the issue slots bound it, 40 us.
//            32 columns: the loads, whose latency 110 warps do not hide);
//   loss     loss[e] += sum of the member's block partials, in block order (the
//            epoch loss accumulates over the batches in stream order);
//   weights  sum over the reduction splits, in split order, of the weights of every
//            layer (the biases between them are the column sums); four parameters per
//            thread, every block size a multiple of 16.
// 4,096 rows, 4 members: 61 + 6 + 11 us in six launches, 23 in one.
constexpr int kRedThreads = 128, kColWarps = kRedThreads / 32, kColsPerWarp = 8;
struct MlpReduce {
  MlpDims d;
  int B, ldT, col_blocks, n_loss, used;
  const __nv_bfloat16* dYT;  // [members][out_pad][ldT]
  const __nv_bfloat16* dZT;  // [layer][members][H][ldT]
  int64_t sLayer;            // between the layers of dZT
  const float* loss_part;    // [members][n_loss]
  float* loss;
  const float* part;  // [split][members][n_params]
  int64_t sSplit;
  float* out;  // [members][n_params]
};
__global__ void __launch_bounds__(kRedThreads) mlp_reduce_kernel(const MlpReduce a) {
  __shared__ uint4 stage[kColWarps][kColsPerWarp][33];
  __shared__ float lpart[1024];
  const MlpDims& d = a.d;
  const int e = blockIdx.y, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if ((int)blockIdx.x < a.col_blocks) {
    const int n0 = (blockIdx.x * kColWarps + warp) * kColsPerWarp, total = d.out_pad + 3 * d.H;
    if (n0 >= total) return;
    // column n0 + j (every layer's columns are a multiple of kColsPerWarp: one layer per warp)
    const __nv_bfloat16* rows;
    int64_t off;
    if (n0 < d.out_pad) {
      rows = a.dYT + ((int64_t)e * d.out_pad + n0) * a.ldT;
      off = d.off_b4 + n0;
    } else {
      const int layer = (n0 - d.out_pad) / d.H, n = n0 - d.out_pad - layer * d.H;
      rows = a.dZT + layer * a.sLayer + ((int64_t)e * d.H + n) * a.ldT;
      off = (layer == 0 ? d.off_b1 : layer == 1 ? d.off_b2 : d.off_b3) + n;
    }
    const int groups = a.B / 256, mine = lane / (32 / kColsPerWarp);
    float s = 0.0f;
    uint4 nxt[kColsPerWarp];
    auto load = [&](int gq) {
#pragma unroll
      for (int j = 0; j < kColsPerWarp; ++j)
        nxt[j] = reinterpret_cast<const uint4*>(rows + (int64_t)j * a.ldT)[gq * 32 + lane];
    };
    if (groups) load(0);
    for (int gq = 0; gq < groups; ++gq) {
#pragma unroll
      for (int j = 0; j < kColsPerWarp; ++j) stage[warp][j][lane] = nxt[j];
      __syncwarp();
      if (gq + 1 < groups) load(gq + 1);
#pragma unroll 8
      for (int j = 0; j < 32; ++j) {
        const uint4 p = stage[warp][mine][j];
        const uint32_t w[4] = {p.x, p.y, p.z, p.w};
#pragma unroll
        for (int q = 0; q < 4; ++q) {  // two BF16 values, the first in the low half
          s += __uint_as_float(w[q] << 16);
          s += __uint_as_float(w[q] & 0xffff0000u);
        }
      }
      __syncwarp();
    }
    for (int i = groups * 256; i < a.B; ++i) s += __bfloat162float(rows[(int64_t)mine * a.ldT + i]);
    if (lane % (32 / kColsPerWarp) == 0) a.out[e * d.n_params + off + mine] = s;
    return;
  }
  if ((int)blockIdx.x == a.col_blocks) {
    float t = 0.0f;
    for (int b0 = 0; b0 < a.n_loss; b0 += 1024) {
      const int nb = min(1024, a.n_loss - b0);
      for (int b = threadIdx.x; b < nb; b += blockDim.x) lpart[b] = a.loss_part[e * a.n_loss + b0 + b];
      __syncthreads();
      if (threadIdx.x == 0) {
#pragma unroll 16
        for (int b = 0; b < nb; ++b) t += lpart[b];
      }
      __syncthreads();
    }
    if (threadIdx.x == 0) a.loss[e] += t;
    return;
  }
  const int64_t i = 4 * ((int64_t)(blockIdx.x - a.col_blocks - 1) * kRedThreads + threadIdx.x);
  if (i >= d.off_b4 || (i >= d.off_b1 && i < d.off_w2) || (i >= d.off_b2 && i < d.off_w3) ||
      (i >= d.off_b3 && i < d.off_w4))
    return;
  const float* p = a.part + e * d.n_params + i;
  float4 acc = {0.0f, 0.0f, 0.0f, 0.0f};
#pragma unroll 8
  for (int sp = 0; sp < a.used; ++sp) {
    const float4 v = *(const float4*)(p + sp * a.sSplit);
    acc.x += v.x;
    acc.y += v.y;
    acc.z += v.z;
    acc.w += v.w;
  }
  *(float4*)(a.out + e * d.n_params + i) = acc;
}

// Adam, and the BF16 copies of the new weights as stored and transposed: a
// block takes a 32 x 32 tile of a weight matrix, which it turns through shared
// memory, or the biases (the last block).  4 members: 7 + 9 us in two launches, the second
// writing every value to its own line, 9 in one.
struct MlpAdam {
  float lr, b1, b2, eps, c1, c2;
};
inline int mlp_tiles(int64_t rows, int64_t cols) { return (int)((rows + 31) / 32 * ((cols + 31) / 32)); }
__global__ void __launch_bounds__(256) mlp_adam_kernel(MlpDims d, float* P, const float* G, float* m, float* v,
                                                       __nv_bfloat16* Ph, __nv_bfloat16* PhT, MlpAdam o) {
  __shared__ __nv_bfloat16 tile[32][34];
  const int64_t base = blockIdx.y * d.n_params;
  auto update = [&](int64_t i) {
    const float g = G[i];
    const float mi = o.b1 * m[i] + (1.0f - o.b1) * g;
    const float vi = o.b2 * v[i] + (1.0f - o.b2) * g * g;
    m[i] = mi;
    v[i] = vi;
    const float p = P[i] - o.lr * (mi * o.c1) / (sqrtf(vi * o.c2) + o.eps);
    P[i] = p;
    const __nv_bfloat16 h = __float2bfloat16(p);
    Ph[i] = h;
    return h;
  };
  const int64_t offs[4] = {d.off_w1, d.off_w2, d.off_w3, d.off_w4};
  const int nr[4] = {d.in_pad, d.H, d.H, d.H}, nc[4] = {d.H, d.H, d.H, d.out_pad};
  int b = blockIdx.x;
#pragma unroll
  for (int l = 0; l < 4; ++l) {
    const int R = nr[l], C = nc[l], tc = (C + 31) / 32, n = (R + 31) / 32 * tc;
    if (b >= n) {
      b -= n;
      continue;
    }
    const int r0 = b / tc * 32, c0 = b % tc * 32, x = threadIdx.x & 31, y = threadIdx.x >> 5;
    for (int r = y; r < 32; r += 8)
      if (r0 + r < R && c0 + x < C) tile[r][x] = update(base + offs[l] + (int64_t)(r0 + r) * C + c0 + x);
    __syncthreads();
    for (int c = y; c < 32; c += 8)
      if (r0 + x < R && c0 + c < C) PhT[base + offs[l] + (int64_t)(c0 + c) * R + r0 + x] = tile[x][c];
    return;
  }
  const int64_t boff[4] = {d.off_b1, d.off_b2, d.off_b3, d.off_b4};
#pragma unroll
  for (int l = 0; l < 4; ++l)
    for (int q = threadIdx.x; q < nc[l]; q += blockDim.x) PhT[base + boff[l] + q] = update(base + boff[l] + q);
}

// ensemble combination in standardised units -> caller units
// Targets are learnt as z = (asinh(y / c) - m) / s (c = 0: z = (y - m) / s);
// the predictive mean and variance map back through y = c sinh(m + s z)
// (delta method for the variance).
// A block takes a few rows and its threads their (row, statistic) pairs, so the
// outputs of the members are read coalesced and every lane has work.  OUT =
// double: the caller's mean and variance, bound by the FP64 pipe (sinh and
// cosh); float: the screen's, rounded once, as sums of two floats with FP64 only
// next to a rounding boundary (the same floats).  65,536 rows x 53 statistics with the
// asinh transform: 0.34 ms in FP64, 0.055 in two floats.
constexpr int kCombinePairs = 2048;  // (row, statistic) pairs per block
template <typename OUT>
__global__ void __launch_bounds__(256) mlp_combine_kernel(const float* __restrict__ Y, int N, int K, int out_pad,
                                                          int members, int64_t sY, int rows_per_block,
                                                          const float* __restrict__ ymean,
                                                          const float* __restrict__ ystd,
                                                          const float* __restrict__ yscale, OUT* __restrict__ mean_out,
                                                          OUT* __restrict__ var_out, double* __restrict__ disagree,
                                                          int aleatoric_only) {
  __shared__ float worst[kCombinePairs];
  const int i0 = blockIdx.x * rows_per_block;
  const int rows = min(rows_per_block, N - i0);
  for (int q = threadIdx.x; q < rows * K; q += blockDim.x) {
    const int i = q / K, k = q - i * K;
    const float* y = Y + (int64_t)(i0 + i) * out_pad + k;
    float mu = 0.0f, mu2 = 0.0f, ale = 0.0f;
    for (int e = 0; e < members; ++e) {
      const float a = y[e * sY];
      const float lv = fminf(fmaxf(y[e * sY + K], kLvMin), kLvMax);
      mu += a;
      mu2 += a * a;
      ale += __expf(lv);
    }
    const float inv = 1.0f / (float)members;
    mu *= inv;
    const float epi = fmaxf(mu2 * inv - mu * mu, 0.0f);
    ale *= inv;
    const float var = aleatoric_only ? ale : ale + epi;
    worst[q] = sqrtf(epi / fmaxf(ale, 1e-12f));
    const int64_t o = (int64_t)i0 * K + q;
    if (sizeof(OUT) == sizeof(float) && mean_out && var_out) {
      float m32, v32;
      if (unscale32(mu, var, ystd[k], ymean[k], yscale ? yscale[k] : 0.0f, m32, v32)) {
        mean_out[o] = (OUT)m32;
        var_out[o] = (OUT)v32;
        continue;
      }
    }
    const double sd = (double)ystd[k];
    const double u = (double)mu * sd + (double)ymean[k];
    const double vu = (double)var * sd * sd;
    const double c = yscale ? (double)yscale[k] : 0.0;
    if (c > 0.0) {
      const double ch = c * cosh(u);
      if (mean_out) mean_out[o] = (OUT)(c * sinh(u));
      if (var_out) var_out[o] = (OUT)(ch * ch * vu);
    } else {
      if (mean_out) mean_out[o] = (OUT)u;
      if (var_out) var_out[o] = (OUT)vu;
    }
  }
  if (!disagree) return;
  __syncthreads();
  for (int i = threadIdx.x; i < rows; i += blockDim.x) {
    float w = 0.0f;
    for (int k = 0; k < K; ++k) w = fmaxf(w, worst[i * K + k]);
    disagree[i0 + i] = w;
  }
}

// ---------------------------------------------------------------------------
// launchers
// ---------------------------------------------------------------------------
static int blocks_for(int64_t n, int t) { return (int)std::min<int64_t>((n + t - 1) / t, 65536); }

// BF16 copies of the parameters: as stored (for dX = dZ W^T) and transposed
// (for the forward GEMMs)
cudaError_t mlp_refresh_bf16(const MlpDims& d, int members, const float* P, __nv_bfloat16* Ph, __nv_bfloat16* PhT,
                             cudaStream_t s) {
  const int64_t n = d.n_params * members;
  mlp_to_bf16_kernel<<<blocks_for(n, 256), 256, 0, s>>>(P, Ph, n);
  mlp_weights_t_kernel<<<blocks_for(n, 256), 256, 0, s>>>(P, d, members, PhT);
  return cudaGetLastError();
}

cudaError_t mlp_init(const MlpDims& d, int members, uint64_t seed, float* P, __nv_bfloat16* Ph, __nv_bfloat16* PhT,
                     cudaStream_t s) {
  const int64_t n = d.n_params * members;
  mlp_init_kernel<<<blocks_for(n, 256), 256, 0, s>>>(d, members, seed, P);
  return mlp_refresh_bf16(d, members, P, Ph, PhT, s);
}

cudaError_t mlp_gather(const float* xn, const float* yn, int64_t N, const MlpDims& d, int B, int64_t base,
                       const uint64_t* perm_ab, int members, __nv_bfloat16* X0, __nv_bfloat16* X0T, int ldT, float* T,
                       cudaStream_t s) {
  dim3 grid((B + kGatherRows - 1) / kGatherRows, members);
  mlp_gather_kernel<<<grid, 256, 0, s>>>(xn, yn, N, d.in_pad, d.K, B, base, perm_ab, X0, X0T, ldT, T,
                                          (int64_t)B * d.in_pad, (int64_t)B * d.K);
  return cudaGetLastError();
}

// Forward pass of all members for B rows.  X0: [members or 1][B][in_pad] (sX = 0:
// one input for every member).  Z: [members][3][B][H] fp32 (may be null), Ah:
// [members][3][B][H] bf16, AhT: [members][3][H][ldT] (transposed activations
// for the weight gradients; null for inference), Y: [members][B][out_pad].
cudaError_t mlp_forward(const MlpDims& d, int members, int B, const __nv_bfloat16* X0, int64_t sX,
                        const __nv_bfloat16* WhT, const float* Pf, float* Z, __nv_bfloat16* Ah, __nv_bfloat16* AhT,
                        int ldT, float* Y, int* err, int sms, cudaStream_t s) {
  if (Z && AhT && sX && mlp_infer_fits(d))
    return mlp_train_forward(d, members, B, X0, WhT, Pf, Z, AhT, ldT, Y, err, sms, s);
  const int H = d.H;
  const int64_t sZ = 3 * (int64_t)B * H, sL = (int64_t)B * H, sLT = (int64_t)H * ldT;
  const int64_t w_off[4] = {d.off_w1, d.off_w2, d.off_w3, d.off_w4};
  const int64_t b_off[4] = {d.off_b1, d.off_b2, d.off_b3, d.off_b4};
  cudaError_t e;
  for (int layer = 0; layer < 4; ++layer) {
    const int K = layer == 0 ? d.in_pad : H;
    const int N = layer == 3 ? d.out_pad : H;
    TcOperand A, Bw;
    A.ptr = layer == 0 ? X0 : Ah + (layer - 1) * sL;
    A.ld = K;
    A.rows = B;
    A.member_stride = layer == 0 ? sX : sZ;
    Bw.ptr = WhT + w_off[layer];   // W^T [N][K]
    Bw.ld = K;
    Bw.rows = N;
    Bw.member_stride = d.n_params;
    TcGemm g{};
    g.M = B;
    g.N = N;
    g.K = K;
    g.k_split = 1;
    g.a_shared = (layer == 0 && sX == 0) ? 1 : 0;
    g.bias = Pf + b_off[layer];
    g.sBias = d.n_params;
    g.err = err;
    if (layer < 3) {
      g.outf = Z ? Z + layer * sL : nullptr;
      g.sOutf = sZ;
      g.ldf = H;
      g.outh = Ah + layer * sL;
      g.sOuth = sZ;
      g.ldh = H;
      g.outhT = AhT ? AhT + layer * sLT : nullptr;
      g.sOuthT = 3 * sLT;
      g.ldhT = ldT;
      e = mlp_tc_gemm(EPI_HIDDEN, A, Bw, g, members, s);
    } else {
      g.outf = Y;
      g.sOutf = (int64_t)B * d.out_pad;
      g.ldf = d.out_pad;
      e = mlp_tc_gemm(EPI_LINEAR, A, Bw, g, members, s);
    }
    if (e != cudaSuccess) return e;
  }
  return cudaSuccess;
}

// Backward pass: dY (bf16 [members][B][out_pad]) and dY^T ([members][out_pad][ldT])
// -> parameter gradients Gf (fp32, every entry written).  dW_l = A_{l-1}^T dZ_l from the
// transposed copies (reduction over the batch split across CTAs, each split
// writing its own slice of Gpart, the slices summed in split order so that a
// training run is reproducible bit for bit); dZ_l = (dZ_{l+1} W_{l+1}^T)
// silu'(Z_l) with its transposed copy.
cudaError_t mlp_backward(const MlpDims& d, int members, int B, const __nv_bfloat16* X0T, const __nv_bfloat16* Wh,
                         float* Z, const __nv_bfloat16* AhT, const __nv_bfloat16* dY, const __nv_bfloat16* dYT,
                         __nv_bfloat16* dZa, __nv_bfloat16* dZb, __nv_bfloat16* dZT, int ldT, float* Gf, float* Gpart,
                         float* loss, const float* loss_part, int* err, int sms, cudaStream_t s) {
  const int H = d.H;
  const int64_t sZ = 3 * (int64_t)B * H, sL = (int64_t)B * H, sLT = (int64_t)H * ldT, sP = d.n_params;
  const int splits = mlp_wgrad_splits(B);
  const int nk = (B + 63) / 64, per = (nk + splits - 1) / splits;
  const int used = (nk + per - 1) / per;  // splits that receive reduction chunks
  cudaError_t e;
  // dW4 = A3^T dY (M = H, N = out_pad), dW_l = A_{l-1}^T dZ_l (M = in_l, N = H)
  TcOperand wa[kWgradGemms], wb[kWgradGemms];
  TcGemm wg[kWgradGemms];
  int n_wg = 0;
  auto wgrad = [&](const TcOperand& A, const TcOperand& Bg, int M, int N, int64_t off) {
    TcGemm g{};
    g.M = M;
    g.N = N;
    g.K = B;
    g.k_split = splits;
    g.outf = Gpart + off;
    g.sOutf = sP;
    g.sSplit = sP * members;
    g.ldf = N;
    g.err = err;
    wa[n_wg] = A;
    wb[n_wg] = Bg;
    wg[n_wg++] = g;
  };
  wgrad(TcOperand{AhT + 2 * sLT, ldT, H, 3 * sLT}, TcOperand{dYT, ldT, d.out_pad, (int64_t)d.out_pad * ldT}, H,
        d.out_pad, d.off_w4);
  const __nv_bfloat16* grad_in = dY;
  int64_t s_gin = (int64_t)B * d.out_pad;
  int ld_gin = d.out_pad;
  const int64_t w_next[3] = {d.off_w2, d.off_w3, d.off_w4};
  const int64_t w_off[3] = {d.off_w1, d.off_w2, d.off_w3};
  __nv_bfloat16* bufs[2] = {dZa, dZb};
  const bool fused = mlp_infer_fits(d);
  if (fused && (e = mlp_train_backward(d, members, B, dY, Wh, Z, dZT, ldT, err, sms, s))) return e;
  for (int layer = 2; layer >= 0; --layer) {
    __nv_bfloat16* dZ = bufs[layer & 1];
    __nv_bfloat16* dZTl = dZT + layer * members * sLT;
    if (!fused) {
      // dZ_l = (grad_in W_{l+1}^T) silu'(Z_l): W_{l+1} stored [H][out] is the K-major [N = H][K = out] operand
      const int Kn = layer == 2 ? d.out_pad : H;
      TcOperand A{grad_in, ld_gin, B, s_gin};
      TcOperand Bw{Wh + w_next[layer], Kn, H, sP};
      TcGemm g{};
      g.M = B;
      g.N = H;
      g.K = Kn;
      g.k_split = 1;
      g.zprev = Z + layer * sL;
      g.sZ = sZ;
      g.ldz = H;
      g.outh = dZ;
      g.sOuth = sL;
      g.ldh = H;
      g.outhT = dZTl;
      g.sOuthT = sLT;
      g.ldhT = ldT;
      g.err = err;
      if ((e = mlp_tc_gemm(EPI_DSILU, A, Bw, g, members, s))) return e;
    }
    const int Min = layer == 0 ? d.in_pad : H;
    wgrad(layer == 0 ? TcOperand{X0T, ldT, d.in_pad, (int64_t)d.in_pad * ldT}
                     : TcOperand{AhT + (layer - 1) * sLT, ldT, H, 3 * sLT},
          TcOperand{dZTl, ldT, H, sLT}, Min, H, w_off[layer]);
    grad_in = dZ;
    s_gin = sL;
    ld_gin = H;
  }
  if ((e = mlp_tc_wgrads(wa, wb, wg, members, s))) return e;
  MlpReduce r{};
  r.d = d;
  r.B = B;
  r.ldT = ldT;
  r.col_blocks = (d.out_pad + 3 * H + kColWarps * kColsPerWarp - 1) / (kColWarps * kColsPerWarp);
  r.n_loss = mlp_loss_blocks(B, d.out_pad);
  r.used = used;
  r.dYT = dYT;
  r.dZT = dZT;
  r.sLayer = members * sLT;
  r.loss_part = loss_part;
  r.loss = loss;
  r.part = Gpart;
  r.sSplit = sP * members;
  r.out = Gf;
  const int wblocks = (int)((d.n_params / 4 + kRedThreads - 1) / kRedThreads);
  mlp_reduce_kernel<<<dim3(r.col_blocks + 1 + wblocks, members), kRedThreads, 0, s>>>(r);
  return cudaGetLastError();
}

cudaError_t mlp_loss(const MlpDims& d, int members, int B, int valid_rows, const float* Y, const float* T,
                     __nv_bfloat16* dY, __nv_bfloat16* dYT, int ldT, float* loss_part, cudaStream_t s) {
  const float inv = 1.0f / (float)(std::max(1, valid_rows) * d.K);
  const int nb = mlp_loss_blocks(B, d.out_pad);
  const int tiles = (B + kLossRows - 1) / kLossRows;
  const size_t smem = (size_t)kLossRows * (d.out_pad + 2) * sizeof(__nv_bfloat16);
  mlp_loss_kernel<<<dim3((nb + kLossBlocks - 1) / kLossBlocks + tiles, members), 256, smem, s>>>(Y, T, B, d.K, d.out_pad, inv, dY, dYT, ldT, loss_part, nb,
                                                              (int64_t)B * d.out_pad, (int64_t)B * d.K);
  return cudaGetLastError();
}

cudaError_t mlp_adam(const MlpDims& d, int members, float* P, const float* G, float* m, float* v,
                     __nv_bfloat16* Ph, __nv_bfloat16* PhT, float lr, int step, cudaStream_t s) {
  const float b1 = 0.9f, b2 = 0.999f, eps = 1e-8f;
  const float c1 = 1.0f / (1.0f - powf(b1, (float)step));
  const float c2 = 1.0f / (1.0f - powf(b2, (float)step));
  const int tiles = mlp_tiles(d.in_pad, d.H) + 2 * mlp_tiles(d.H, d.H) + mlp_tiles(d.H, d.out_pad);
  mlp_adam_kernel<<<dim3(tiles + 1, members), 256, 0, s>>>(d, P, G, m, v, Ph, PhT, MlpAdam{lr, b1, b2, eps, c1, c2});
  return cudaGetLastError();
}

template <typename OUT>
static cudaError_t combine(const MlpDims& d, int members, int N, const float* Y, const float* ymean,
                           const float* ystd, const float* yscale, OUT* mean_out, OUT* var_out, double* disagree,
                           int aleatoric_only, cudaStream_t s) {
  const int rows = std::max(1, kCombinePairs / d.K);
  mlp_combine_kernel<OUT><<<(N + rows - 1) / rows, 256, 0, s>>>(Y, N, d.K, d.out_pad, members, (int64_t)N * d.out_pad,
                                                                rows, ymean, ystd, yscale, mean_out, var_out, disagree,
                                                                aleatoric_only);
  return cudaGetLastError();
}

cudaError_t mlp_combine(const MlpDims& d, int members, int N, const float* Y, const float* ymean, const float* ystd,
                        const float* yscale, double* mean_out, double* var_out, double* disagree, int aleatoric_only,
                        cudaStream_t s) {
  return combine<double>(d, members, N, Y, ymean, ystd, yscale, mean_out, var_out, disagree, aleatoric_only, s);
}

cudaError_t mlp_combine32(const MlpDims& d, int members, int N, const float* Y, const float* ymean,
                          const float* ystd, const float* yscale, float* mean_out, float* var_out, double* disagree,
                          cudaStream_t s) {
  return combine<float>(d, members, N, Y, ymean, ystd, yscale, mean_out, var_out, disagree, 0, s);
}

}  // namespace abc
