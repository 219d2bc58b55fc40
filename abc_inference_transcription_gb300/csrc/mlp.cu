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

__global__ void __launch_bounds__(256) mlp_loss_kernel(const float* Y, const float* T, int B, int K, int out_pad,
                                                       float inv_count, __nv_bfloat16* dY, __nv_bfloat16* dYT, int ldT,
                                                       float* loss_part, int64_t sY, int64_t sT) {
  const int e = blockIdx.y;
  float local = 0.0f;
  for (int idx = blockIdx.x * blockDim.x + threadIdx.x; idx < B * out_pad; idx += gridDim.x * blockDim.x) {
    const int i = idx / out_pad, c = idx - (idx / out_pad) * out_pad;
    float grad = 0.0f;
    if (c < K) {
      const float t = T[e * sT + (int64_t)i * K + c];
      if (t == t) {
        const float mu = Y[e * sY + (int64_t)i * out_pad + c];
        const float lv_raw = Y[e * sY + (int64_t)i * out_pad + K + c];
        const float lv = fminf(fmaxf(lv_raw, kLvMin), kLvMax);
        const float r = t - mu;
        const float ei = __expf(-lv);
        local += 0.5f * (lv + r * r * ei);
        grad = -r * ei * inv_count;
      }
    } else if (c < 2 * K) {
      const float t = T[e * sT + (int64_t)i * K + (c - K)];
      if (t == t) {
        const float mu = Y[e * sY + (int64_t)i * out_pad + (c - K)];
        const float lv_raw = Y[e * sY + (int64_t)i * out_pad + c];
        const bool inside = lv_raw > kLvMin && lv_raw < kLvMax;
        const float lv = fminf(fmaxf(lv_raw, kLvMin), kLvMax);
        const float r = t - mu;
        grad = inside ? 0.5f * (1.0f - r * r * __expf(-lv)) * inv_count : 0.0f;
      }
    }
    const __nv_bfloat16 gb = __float2bfloat16(grad);
    dY[e * sY + idx] = gb;
    dYT[(int64_t)e * out_pad * ldT + (int64_t)c * ldT + i] = gb;
  }
  // block sum in a fixed order: warps by shuffles, then warp 0 over the warp sums
  __shared__ float wsum[8];
  for (int o = 16; o > 0; o >>= 1) local += __shfl_xor_sync(0xffffffffu, local, o);
  if ((threadIdx.x & 31) == 0) wsum[threadIdx.x >> 5] = local;
  __syncthreads();
  if (threadIdx.x == 0) {
    float t = 0.0f;
    for (int w = 0; w < (int)(blockDim.x >> 5); ++w) t += wsum[w];
    loss_part[e * gridDim.x + blockIdx.x] = t * inv_count;
  }
}

// loss[e] += sum of the member's block partials, in block order (the epoch
// loss accumulates over the batches in stream order).  The chain of additions
// reads shared memory: from global memory 1,024 partials took 25 us.
__global__ void __launch_bounds__(1024) mlp_loss_sum_kernel(const float* loss_part, int n_blocks, float* loss) {
  __shared__ float part[1024];
  const int e = blockIdx.x;
  float t = 0.0f;
  for (int b0 = 0; b0 < n_blocks; b0 += 1024) {
    const int nb = min(1024, n_blocks - b0);
    if ((int)threadIdx.x < nb) part[threadIdx.x] = loss_part[e * n_blocks + b0 + threadIdx.x];
    __syncthreads();
    if (threadIdx.x == 0) {
#pragma unroll 16
      for (int b = 0; b < nb; ++b) t += part[b];
    }
    __syncthreads();
  }
  if (threadIdx.x == 0) loss[e] += t;
}

// out[z][i] = sum over the used reduction splits of part[split][z][i], in split
// order, for the weights of every layer (the biases between them are column
// sums); four parameters per thread, every block size a multiple of 16
__global__ void __launch_bounds__(256) mlp_split_sum_kernel(const float* part, int used, int64_t sSplit, MlpDims d,
                                                            float* out) {
  const int z = blockIdx.y;
  for (int64_t i = 4 * ((int64_t)blockIdx.x * blockDim.x + threadIdx.x); i < d.n_params;
       i += 4 * (int64_t)gridDim.x * blockDim.x) {
    if ((i >= d.off_b1 && i < d.off_w2) || (i >= d.off_b2 && i < d.off_w3) || (i >= d.off_b3 && i < d.off_w4) ||
        i >= d.off_b4)
      continue;
    const float* p = part + z * d.n_params + i;
    float4 acc = {0.0f, 0.0f, 0.0f, 0.0f};
#pragma unroll 4
    for (int sp = 0; sp < used; ++sp) {
      const float4 v = *(const float4*)(p + sp * sSplit);
      acc.x += v.x;
      acc.y += v.y;
      acc.z += v.z;
      acc.w += v.w;
    }
    *(float4*)(out + z * d.n_params + i) = acc;
  }
}

// db[n] = sum_i dZ[i][n] for every member, in row order (a training run is
// reproducible bit for bit, and independent of the launch), from the transposed
// copy [n][ldT].  The additions are one chain per column, so a warp takes a
// column: its lanes load 256 rows at once (coalesced, the next 256 in flight) and
// pass them through shared memory to the chain.  4,096 rows: 15 us, against
// 39 with a lane per column and 266 down dZ's columns.
constexpr int kColWarps = 4;
__global__ void __launch_bounds__(32 * kColWarps) mlp_colsum_kernel(const __nv_bfloat16* dZT, int B, int N, int ldT,
                                                                    int64_t sZT, float* db, int64_t sDb) {
  __shared__ uint4 stage[kColWarps][32];
  const int e = blockIdx.y, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int n = blockIdx.x * kColWarps + warp;
  if (n >= N) return;
  const __nv_bfloat16* row = dZT + e * sZT + (int64_t)n * ldT;
  const uint4* src = reinterpret_cast<const uint4*>(row);
  const int groups = B / 256;
  float s = 0.0f;
  uint4 nxt = {0u, 0u, 0u, 0u};
  if (groups) nxt = src[lane];
  for (int gq = 0; gq < groups; ++gq) {
    stage[warp][lane] = nxt;
    __syncwarp();
    if (gq + 1 < groups) nxt = src[(gq + 1) * 32 + lane];
#pragma unroll 8
    for (int j = 0; j < 32; ++j) {
      const uint4 p = stage[warp][j];
      const uint32_t w[4] = {p.x, p.y, p.z, p.w};
#pragma unroll
      for (int q = 0; q < 4; ++q) {  // two BF16 values, the first in the low half
        s += __uint_as_float(w[q] << 16);
        s += __uint_as_float(w[q] & 0xffff0000u);
      }
    }
    __syncwarp();
  }
  for (int i = groups * 256; i < B; ++i) s += __bfloat162float(row[i]);
  if (lane == 0) db[e * sDb + n] = s;
}

__global__ void mlp_adam_kernel(float* P, const float* G, float* m, float* v, __nv_bfloat16* Ph, int64_t n, float lr,
                                float b1, float b2, float eps, float c1, float c2) {
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
    const float g = G[i];
    const float mi = b1 * m[i] + (1.0f - b1) * g;
    const float vi = b2 * v[i] + (1.0f - b2) * g * g;
    m[i] = mi;
    v[i] = vi;
    const float p = P[i] - lr * (mi * c1) / (sqrtf(vi * c2) + eps);
    P[i] = p;
    Ph[i] = __float2bfloat16(p);
  }
}

// ensemble combination in standardised units -> caller units
// Targets are learnt as z = (asinh(y / c) - m) / s (c = 0: z = (y - m) / s);
// the predictive mean and variance map back through y = c sinh(m + s z)
// (delta method for the variance).
// A block takes a few rows and its threads their (row, statistic) pairs, so the
// outputs of the members are read coalesced and every lane of the FP64 pipe,
// which bounds this (sinh and cosh), has work.  OUT = double: the caller's
// mean and variance; float: the screen's, rounded once.  65,536 rows x 53
// statistics with the asinh transform: 0.36 ms, 0.46 with a thread per row.
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
    const double sd = (double)ystd[k];
    const double u = (double)mu * sd + (double)ymean[k];
    const double vu = (double)var * sd * sd;
    const double c = yscale ? (double)yscale[k] : 0.0;
    const int64_t o = (int64_t)i0 * K + q;
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
                        int ldT, float* Y, int* err, cudaStream_t s) {
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
                         const float* Z, const __nv_bfloat16* AhT, const __nv_bfloat16* dY, const __nv_bfloat16* dYT,
                         __nv_bfloat16* dZa, __nv_bfloat16* dZb, __nv_bfloat16* dZTa, __nv_bfloat16* dZTb, int ldT,
                         float* Gf, float* Gpart, int* err, cudaStream_t s) {
  const int H = d.H;
  const int64_t sZ = 3 * (int64_t)B * H, sL = (int64_t)B * H, sLT = (int64_t)H * ldT, sP = d.n_params;
  const int splits = mlp_wgrad_splits(B);
  const int nk = (B + 63) / 64, per = (nk + splits - 1) / splits;
  const int used = (nk + per - 1) / per;  // splits that receive reduction chunks
  cudaError_t e;
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
    return mlp_tc_gemm(EPI_PARTIAL, A, Bg, g, members, s);
  };
  // layer 4: dW4 = A3^T dY (M = H, N = out_pad), db4 = colsum(dY)
  {
    TcOperand A{AhT + 2 * sLT, ldT, H, 3 * sLT};
    TcOperand Bg{dYT, ldT, d.out_pad, (int64_t)d.out_pad * ldT};
    if ((e = wgrad(A, Bg, H, d.out_pad, d.off_w4))) return e;
    mlp_colsum_kernel<<<dim3((d.out_pad + kColWarps - 1) / kColWarps, members), 32 * kColWarps, 0, s>>>(
        dYT, B, d.out_pad, ldT, (int64_t)d.out_pad * ldT, Gf + d.off_b4, sP);
  }
  const __nv_bfloat16* grad_in = dY;
  int64_t s_gin = (int64_t)B * d.out_pad;
  int ld_gin = d.out_pad;
  const int64_t w_next[3] = {d.off_w2, d.off_w3, d.off_w4};
  const int64_t b_off[3] = {d.off_b1, d.off_b2, d.off_b3};
  const int64_t w_off[3] = {d.off_w1, d.off_w2, d.off_w3};
  __nv_bfloat16* bufs[2] = {dZa, dZb};
  __nv_bfloat16* bufsT[2] = {dZTa, dZTb};
  for (int layer = 2; layer >= 0; --layer) {
    __nv_bfloat16* dZ = bufs[layer & 1];
    __nv_bfloat16* dZT = bufsT[layer & 1];
    {
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
      g.outhT = dZT;
      g.sOuthT = sLT;
      g.ldhT = ldT;
      g.err = err;
      if ((e = mlp_tc_gemm(EPI_DSILU, A, Bw, g, members, s))) return e;
    }
    {
      // dW_l = A_{l-1}^T dZ_l (M = in_l, N = H), db_l = colsum(dZ_l)
      const int Min = layer == 0 ? d.in_pad : H;
      TcOperand A = layer == 0 ? TcOperand{X0T, ldT, d.in_pad, (int64_t)d.in_pad * ldT}
                               : TcOperand{AhT + (layer - 1) * sLT, ldT, H, 3 * sLT};
      TcOperand Bg{dZT, ldT, H, sLT};
      if ((e = wgrad(A, Bg, Min, H, w_off[layer]))) return e;
      mlp_colsum_kernel<<<dim3((H + kColWarps - 1) / kColWarps, members), 32 * kColWarps, 0, s>>>(dZT, B, H, ldT, sLT,
                                                                                             Gf + b_off[layer], sP);
    }
    grad_in = dZ;
    s_gin = sL;
    ld_gin = H;
  }
  mlp_split_sum_kernel<<<dim3((unsigned)((d.n_params / 4 + 255) / 256), members), 256, 0, s>>>(
      Gpart, used, sP * members, d, Gf);
  return cudaGetLastError();
}

cudaError_t mlp_loss(const MlpDims& d, int members, int B, int valid_rows, const float* Y, const float* T,
                     __nv_bfloat16* dY, __nv_bfloat16* dYT, int ldT, float* loss, float* loss_part, cudaStream_t s) {
  const float inv = 1.0f / (float)(std::max(1, valid_rows) * d.K);
  const int nb = mlp_loss_blocks(B, d.out_pad);
  mlp_loss_kernel<<<dim3(nb, members), 256, 0, s>>>(Y, T, B, d.K, d.out_pad, inv, dY, dYT, ldT, loss_part,
                                                    (int64_t)B * d.out_pad, (int64_t)B * d.K);
  mlp_loss_sum_kernel<<<members, 1024, 0, s>>>(loss_part, nb, loss);
  return cudaGetLastError();
}

cudaError_t mlp_adam(const MlpDims& d, int members, float* P, const float* G, float* m, float* v,
                     __nv_bfloat16* Ph, __nv_bfloat16* PhT, float lr, int step, cudaStream_t s) {
  const float b1 = 0.9f, b2 = 0.999f, eps = 1e-8f;
  const float c1 = 1.0f / (1.0f - powf(b1, (float)step));
  const float c2 = 1.0f / (1.0f - powf(b2, (float)step));
  const int64_t n = d.n_params * members;
  mlp_adam_kernel<<<blocks_for(n, 256), 256, 0, s>>>(P, G, m, v, Ph, n, lr, b1, b2, eps, c1, c2);
  mlp_weights_t_kernel<<<blocks_for(n, 256), 256, 0, s>>>(P, d, members, PhT);
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
