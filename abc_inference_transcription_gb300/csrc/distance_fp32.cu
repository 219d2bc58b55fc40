// distance_fp32.cu — FP32 particle x gene distance with a fused epilogue
// (candidate emission or subsample export) and the per-gene threshold pass.
// The P x G error matrix is never written in full.
#include <atomic>

#include "distance.cuh"
#include "kernels.h"
#include "smem_attr.h"

namespace abc {

// 256 threads = 16 x 16; thread (tx, ty) owns particles ty + 16 i and genes
// tx + 16 j (i, j < 8) of a 128 x 128 tile.  Statistics stream through shared
// memory kDistKc at a time, stored k-major so one row serves all threads.
//
// GJ genes per thread: 8, or 1 (a tile of 16 genes) for few genes, where the
// wide tile computes mostly padding (32,768 rows x 4 genes of 53 statistics: 35 us wide, 14
// narrow).  The rows are padded by one word: without it the 16 statistics of a
// row go to one bank.
template <int GJ>
__global__ void __launch_bounds__(256) dist_fast_kernel(const float* __restrict__ s32,
                                                        const float* __restrict__ sw,
                                                        const float* __restrict__ dw, int64_t P, int64_t G,
                                                        int K, const float* __restrict__ X, Cand* cand,
                                                        float* cand_e, unsigned long long* n_cand, int64_t cap,
                                                        float* esub, int64_t stride, int64_t n_sub) {
  constexpr int kGenes = 16 * GJ;
  __shared__ float ss[kDistKc][kDistTile + 1];
  __shared__ float sa[kDistKc][kGenes + 1];
  __shared__ float sd[kDistKc][kGenes + 1];
  const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
  const int64_t g0 = (int64_t)blockIdx.x * kGenes;
  const int64_t r0 = (int64_t)blockIdx.y * kDistTile;  // row = particle (emit) or subsample row
  const bool sample = esub != nullptr;
  const int64_t nrows = sample ? n_sub : P;
  float acc[8][GJ];
#pragma unroll
  for (int i = 0; i < 8; ++i)
#pragma unroll
    for (int j = 0; j < GJ; ++j) acc[i][j] = 0.0f;

  for (int k0 = 0; k0 < K; k0 += kDistKc) {
    // cooperative loads: 128 rows x kDistKc values for each of the three tiles
    for (int idx = threadIdx.x; idx < kDistKc * kDistTile; idx += 256) {
      const int r = idx / kDistKc, kk = idx - (idx / kDistKc) * kDistKc;
      const int k = k0 + kk;
      const int64_t row = r0 + r;
      float sv = 0.0f;
      if (row < nrows && k < K) {
        const int64_t p = sample ? row * stride : row;
        sv = s32[p * K + k];
      }
      ss[kk][r] = sv;
      if (r >= kGenes) continue;
      const int64_t g = g0 + r;
      float av = 0.0f, dv = 0.0f;
      if (g < G && k < K) {
        av = sw[g * K + k];
        dv = dw[g * K + k];
      }
      sa[kk][r] = av;
      sd[kk][r] = dv;
    }
    __syncthreads();
    const int kc = (K - k0) < kDistKc ? (K - k0) : kDistKc;
#pragma unroll 4
    for (int kk = 0; kk < kc; ++kk) {
      float s[8], a[GJ], d[GJ];
#pragma unroll
      for (int i = 0; i < 8; ++i) s[i] = ss[kk][ty + 16 * i];
#pragma unroll
      for (int j = 0; j < GJ; ++j) {
        a[j] = sa[kk][tx + 16 * j];
        d[j] = sd[kk][tx + 16 * j];
      }
#pragma unroll
      for (int i = 0; i < 8; ++i)
#pragma unroll
        for (int j = 0; j < GJ; ++j) {
          float t = fmaf(-a[j], s[i], d[j]);
          acc[i][j] = fmaf(t, t, acc[i][j]);
        }
    }
    __syncthreads();
  }
  const float invK = 1.0f / (float)K;
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    const int64_t row = r0 + ty + 16 * i;
    if (row >= nrows) continue;
#pragma unroll
    for (int j = 0; j < GJ; ++j) {
      const int64_t g = g0 + tx + 16 * j;
      if (g >= G) continue;
      float e = fminf(acc[i][j] * invK, 10.0f);
      if (acc[i][j] != acc[i][j]) e = acc[i][j];  // keep NaN (fminf would drop it)
      if (sample) {
        esub[row * G + g] = e;
      } else if (e <= X[g]) {
        unsigned long long slot = atomicAdd(n_cand, 1ull);
        if (slot < (unsigned long long)cap) {
          Cand c;
          c.p = (int32_t)row;
          c.g = (int32_t)g;
          cand[slot] = c;
          if (cand_e) cand_e[slot] = e;
        }
      }
    }
  }
}

cudaError_t launch_dist_fast(const float* s32, const float* sw, const float* dw, int64_t P, int64_t G, int K,
                             const float* X, Cand* cand, float* cand_e, unsigned long long* n_cand, int64_t cap,
                             float* esub, int64_t stride, int64_t n_sub, cudaStream_t s) {
  const int64_t rows = esub ? n_sub : P;
  if (rows <= 0 || G <= 0) return cudaSuccess;
  const int genes = G <= 32 ? 16 : kDistTile;
  dim3 grid((unsigned)((G + genes - 1) / genes), (unsigned)((rows + kDistTile - 1) / kDistTile));
  if (genes == 16)
    dist_fast_kernel<1><<<grid, 256, 0, s>>>(s32, sw, dw, P, G, K, X, cand, cand_e, n_cand, cap, esub, stride, n_sub);
  else
    dist_fast_kernel<8><<<grid, 256, 0, s>>>(s32, sw, dw, P, G, K, X, cand, cand_e, n_cand, cap, esub, stride, n_sub);
  return cudaGetLastError();
}

// Cumulative histogram search shared by the threshold and refinement kernels:
// the first bin at which the running count of hist[0..kHistBins) reaches k
// (-1 if it never does).  Called by every thread of a CTA of at least 256;
// csum is 256 words of shared memory.  The first warp scans the 256 partial
// counts by shuffles and one lane walks the 128 bins that hold the answer.
__device__ int hist_find(const unsigned int* hist, int64_t k, unsigned int* csum) {
  constexpr int per = kHistBins / 256;
  if (threadIdx.x < 256) {
    unsigned int local = 0;
#pragma unroll
    for (int b = 0; b < per; ++b) local += hist[threadIdx.x * per + b];
    csum[threadIdx.x] = local;
  }
  __syncthreads();
  int found = -1;
  if (threadIdx.x < 32) {
    const int lane = threadIdx.x;
    unsigned long long own = 0;
    for (int b = 0; b < 8; ++b) own += csum[lane * 8 + b];
    unsigned long long run = own;
    for (int o = 1; o < 32; o <<= 1) {
      const unsigned long long v = __shfl_up_sync(0xffffffffu, run, o);
      if (lane >= o) run += v;
    }
    const unsigned m = __ballot_sync(0xffffffffu, run >= (unsigned long long)k);
    if (m && lane == __ffs(m) - 1) {
      run -= own;
      for (int c = lane * 8; found < 0; ++c) {
        if (run + csum[c] < (unsigned long long)k) {
          run += csum[c];
          continue;
        }
        for (int b = 0; found < 0; ++b) {
          run += hist[c * per + b];
          if (run >= (unsigned long long)k) found = c * per + b;
        }
      }
    }
    if (m) found = __shfl_sync(0xffffffffu, found, __ffs(m) - 1);
  }
  return found;  // meaningful in the first warp
}

// Histogram of the subsample errors of GB neighbouring genes per CTA on a sqrt
// scale, then per gene the bin where the running count reaches k_sub gives X[g]
// (its upper edge widened by twice the error bound b0_g + b1 e of the candidate
// pass).  The errors lie row by row, so eight genes at a time read whole 32-byte
// sectors; the last bin, where almost all of them fall (the clip), is counted in
// registers instead of by atomics on one word.  32,768 rows: 2,000 genes 0.32
// ms with a CTA of 256 threads per gene, 0.093 now; 4 genes 80 us, 10 now.
__global__ void __launch_bounds__(1024) dist_threshold_kernel(const float* __restrict__ esub, int64_t n_sub,
                                                              int64_t G, int64_t k_sub, int log_gb, const float* b0,
                                                              float b1, float* X) {
  extern __shared__ unsigned int hist[];  // GB x kHistBins
  __shared__ unsigned int csum[256];
  const int GB = 1 << log_gb;
  const int64_t g0 = (int64_t)blockIdx.x * GB;
  for (int b = threadIdx.x; b < GB * kHistBins; b += blockDim.x) hist[b] = 0u;
  __syncthreads();
  const int j = threadIdx.x & (GB - 1);
  unsigned int last = 0;
  if (g0 + j < G) {
    unsigned int* h = hist + j * kHistBins;
    const int64_t step = blockDim.x >> log_gb;
    constexpr int kAhead = 16;  // loads in flight per thread
    for (int64_t r0 = threadIdx.x >> log_gb; r0 < n_sub; r0 += kAhead * step) {
      float e[kAhead];
#pragma unroll
      for (int u = 0; u < kAhead; ++u) {
        const int64_t r = r0 + u * step;
        e[u] = r < n_sub ? __ldg(esub + r * G + g0 + j) : __int_as_float(0x7fc00000);
      }
#pragma unroll
      for (int u = 0; u < kAhead; ++u) {
        if (e[u] >= 10.0f)  // the clip: the last bin
          ++last;
        else if (e[u] == e[u])
          atomicAdd(&h[hist_bin(e[u])], 1u);
      }
    }
    if (last) atomicAdd(&h[kHistBins - 1], last);
  }
  __syncthreads();
  for (int q = 0; q < GB && g0 + q < G; ++q) {
    const int found = hist_find(hist + q * kHistBins, k_sub, csum);
    if (threadIdx.x == 0) {
      float x;
      if (found < 0 || k_sub <= 0) {
        x = INFINITY;
      } else {
        const float bg = b0[g0 + q];
        const float up = hist_upper(found);
        const float xp = up + 1.01f * (bg + b1 * up);
        x = xp + 1.01f * (bg + b1 * xp);
      }
      X[g0 + q] = x;
    }
    __syncthreads();  // csum is rewritten
  }
}

cudaError_t launch_dist_threshold(const float* esub, int64_t n_sub, int64_t G, int64_t k_sub, const float* b0,
                                  float b1, float* X, int sms, cudaStream_t s) {
  if (G <= 0) return cudaSuccess;
  // as many genes per CTA as leave every multiprocessor one, at most 8 (128 KB of histograms)
  int lg = 0;
  while (lg < 3 && (G >> (lg + 1)) >= sms) ++lg;
  const size_t smem = ((size_t)sizeof(unsigned int) * kHistBins) << lg;
  static std::atomic<uint64_t> attr{0};  // devices where the limit is set, shared by all contexts
  cudaError_t e = set_smem_once(attr, dist_threshold_kernel, (int)(sizeof(unsigned int) * kHistBins * 8));
  if (e != cudaSuccess) return e;
  dist_threshold_kernel<<<(unsigned)((G + (1 << lg) - 1) >> lg), 1024, smem, s>>>(esub, n_sub, G, k_sub, lg, b0, b1,
                                                                                 X);
  return cudaGetLastError();
}

// ---------------------------------------------------------------------------
// thresholds of the candidate pass and the refinement before the FP64 recheck
// ---------------------------------------------------------------------------

__global__ void fill_kernel(float* x, int64_t n, float v) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) x[i] = v;
}

cudaError_t launch_fill(float* x, int64_t n, float v, cudaStream_t s) {
  if (n <= 0) return cudaSuccess;
  fill_kernel<<<(unsigned)((n + 255) / 256), 256, 0, s>>>(x, n, v);
  return cudaGetLastError();
}

// X_g for an error threshold e_g (eps, or thr[g]): every pair with err <= e_g
// has a candidate-pass error <= e_g + B_g(e_g) <= X_g = e_g + 2 B_g(e_g)
// (e_g rounded up to FP32 first).  e_g >= 10: every finite pair; e_g < 0: none.
__global__ void x_from_thr_kernel(const double* thr, double eps, int64_t G, const float* b0, float b1, float* X) {
  const int64_t g = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (g >= G) return;
  const double ev = thr ? thr[g] : eps;
  float x;
  if (ev >= 10.0) {
    x = INFINITY;
  } else if (ev < 0.0) {
    x = -1.0f;
  } else {
    const float e = __double2float_ru(ev);
    x = __fadd_ru(e, __fmul_ru(2.0f, __fmaf_ru(b1, e, b0[g])));
  }
  X[g] = x;
}

cudaError_t launch_x_from_thr(const double* thr, double eps, int64_t G, const float* b0, float b1, float* X,
                              cudaStream_t s) {
  if (G <= 0) return cudaSuccess;
  x_from_thr_kernel<<<(unsigned)((G + 255) / 256), 256, 0, s>>>(thr, eps, G, b0, b1, X);
  return cudaGetLastError();
}

// A candidate whose error is certainly above the clip value 10, so that it is 10:
// |e32 - err| <= b0 + b1 err (twice that covers the rounding here).  Only an
// unclipped e32 can say so: the tensor-core pass's, not that of dist_fast_kernel.
__device__ __forceinline__ float sure_clip(float b0, float b1) { return fmaf(2.0f, fmaf(10.0f, b1, b0), 10.0f); }
__device__ __forceinline__ bool surely_clipped(float e, float sure) { return e > sure && e < INFINITY; }

// Histogram of the candidates' FP32 errors per gene (G x kCandBins counters:
// kHistBins of errors, then the surely clipped ones).
constexpr int kCandBins = kHistBins + 1;
__device__ __forceinline__ int cand_bin(float e, float sure) {
  return surely_clipped(e, sure) ? kHistBins : hist_bin(fminf(fmaxf(e, 0.0f), 10.0f));
}
__global__ void cand_hist_kernel(const Cand* cand, const float* e, int64_t n, const float* b0, float b1,
                                 unsigned int* hist) {
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
    const float x = e[i];
    const int32_t g = cand[i].g;
    if (x == x) atomicAdd(&hist[(int64_t)g * kCandBins + cand_bin(x, sure_clip(b0[g], b1))], 1u);
  }
}

// The same with the histograms of all genes in shared memory, for few genes:
// with 4 of them the candidates' global atomics met on a few thousand words (300,000
// candidates: 66 us, 14 here).
constexpr int kSmemHistGenes = 12;  // 192 KB
__global__ void __launch_bounds__(1024) cand_hist_smem_kernel(const Cand* cand, const float* e, int64_t n, int G,
                                                              const float* b0, float b1, unsigned int* hist) {
  extern __shared__ unsigned int sh[];  // G x kCandBins
  __shared__ float sure[kSmemHistGenes];
  if (threadIdx.x < G) sure[threadIdx.x] = sure_clip(b0[threadIdx.x], b1);
  for (int b = threadIdx.x; b < G * kCandBins; b += blockDim.x) sh[b] = 0u;
  __syncthreads();
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
    const float x = e[i];
    const int32_t g = cand[i].g;
    if (x == x) atomicAdd(&sh[g * kCandBins + cand_bin(x, sure[g])], 1u);
  }
  __syncthreads();
  for (int b = threadIdx.x; b < G * kCandBins; b += blockDim.x)
    if (sh[b]) atomicAdd(&hist[b], sh[b]);
}

// Per gene: when at least k candidates have an FP32 error <= a (the upper edge
// of the bin that completes k), k particles have err <= a' = (a + b0)/(1 - b1),
// so the k smallest errors are <= a', and every particle with err <= a' has an
// FP32 error <= a' + B(a').  Xt = a' + 2 B(a') keeps them all and passes the
// acceptance check (Xt - B(Xt) >= a' for b1 <= 1/2).  Xt never exceeds X.
// Only for a' < 10: at the clip value every particle beyond it ties at 10,
// whatever its unclipped error, so no tighter threshold is safe there.  Ties are
// ordered by index, so of the surely clipped candidates only those with an index
// below p_end matter: of the first k + (P - n) + c particles at most P - n are not
// candidates (n are) and at most c candidates are not surely clipped, so k of
// them are, and come before every clipped one from p_end on.  With a cut at 10,
// the top 1 % of 4 x 10^6 particles for two genes rechecks and sorts some 2 x 72,000
// pairs so instead of 8 x 10^6 (2.4 ms for the selection, 113 before).
__global__ void __launch_bounds__(256) refine_kernel(const unsigned int* hist, int64_t P, int64_t G, int64_t k,
                                                     const float* X, const float* b0, float b1, float* Xt,
                                                     float2* cut) {
  __shared__ unsigned int csum[256];
  const int64_t g = blockIdx.x;
  const int found = hist_find(hist + g * kCandBins, k, csum);
  if (threadIdx.x == 0) {
    float x = X[g];
    if (found >= 0 && k > 0) {
      const float a = hist_upper(found);
      if (a < 10.0f) {
        const float bg = b0[g];
        const float a1 = __fdiv_ru(__fadd_ru(a, bg), __fsub_rd(1.0f, b1));
        const float xt = __fadd_ru(a1, __fmul_ru(2.0f, __fmaf_ru(b1, a1, bg)));
        if (a1 < 10.0f && xt < x) x = xt;
      }
    }
    Xt[g] = x;
    int64_t end = P;
    if (x >= 10.0f) {
      int64_t c = 0;
      for (int b = 0; b < 256; ++b) c += csum[b];
      const int64_t cand = c + hist[g * kCandBins + kHistBins];
      end = min(P, k + (P - cand) + c);
    }
    cut[g] = make_float2(sure_clip(b0[g], b1), __int_as_float((int)min(end, (int64_t)INT32_MAX)));
  }
}

// Keep candidates with e <= Xt[g] (e clipped at 10, as the error is) that are not
// surely clipped or have an index below p_end[g] (cut[g]: the bound of sure
// clipping and p_end; looked at only where Xt lets clipped ones pass).  A block takes 4 x 256 candidates per
// iteration and appends its kept ones with one global atomic (positions from
// the warps' ballots), so the shared output counter sees one atomic per 1,024
// candidates instead of one per warp.
constexpr int kFilterItems = 4;
__global__ void __launch_bounds__(256) cand_filter_kernel(const Cand* cand, const float* e, int64_t n, const float* Xt,
                                                          const float2* cut, Cand* out, unsigned long long* count) {
  __shared__ unsigned int wc[kFilterItems * 8];
  __shared__ unsigned long long base;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int64_t per = (int64_t)kFilterItems * blockDim.x;
  for (int64_t i0 = (int64_t)blockIdx.x * per; i0 < n; i0 += (int64_t)gridDim.x * per) {
    bool keep[kFilterItems], tie = false;
    Cand cd[kFilterItems];
    unsigned m[kFilterItems];
#pragma unroll
    for (int j = 0; j < kFilterItems; ++j) {
      const int64_t i = i0 + (int64_t)j * blockDim.x + threadIdx.x;
      keep[j] = false;
      if (i < n) {
        cd[j] = cand[i];
        const float x = e[i], xt = Xt[cd[j].g];
        const bool clip = x > 10.0f && xt >= 10.0f;
        keep[j] = x <= xt || clip;
        tie = tie || clip;
      }
    }
    if (tie) {
#pragma unroll
      for (int j = 0; j < kFilterItems; ++j) {
        if (keep[j]) {
          const float x = e[i0 + (int64_t)j * blockDim.x + threadIdx.x];
          const float2 c = cut[cd[j].g];
          keep[j] = !surely_clipped(x, c.x) || cd[j].p < __float_as_int(c.y);
        }
      }
    }
#pragma unroll
    for (int j = 0; j < kFilterItems; ++j) {
      m[j] = __ballot_sync(0xffffffffu, keep[j]);
      if (lane == 0) wc[j * 8 + warp] = __popc(m[j]);
    }
    __syncthreads();
    if (threadIdx.x == 0) {  // exclusive scan of the 32 warp counts, one reservation
      unsigned int run = 0;
      for (int q = 0; q < kFilterItems * 8; ++q) {
        const unsigned int v = wc[q];
        wc[q] = run;
        run += v;
      }
      base = run ? atomicAdd(count, (unsigned long long)run) : 0ull;
    }
    __syncthreads();
#pragma unroll
    for (int j = 0; j < kFilterItems; ++j)
      if (keep[j]) out[base + wc[j * 8 + warp] + __popc(m[j] & ((1u << lane) - 1u))] = cd[j];
    __syncthreads();  // wc and base are rewritten by the next iteration
  }
}

__global__ void scatter_errors_kernel(const Cand* cand, const float* e, int64_t n, int64_t G, float* out) {
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
    out[(int64_t)cand[i].p * G + cand[i].g] = e[i] > 10.0f ? 10.0f : e[i];
}

cudaError_t launch_scatter_errors(const Cand* cand, const float* e, int64_t n, int64_t G, float* out, cudaStream_t s) {
  if (n <= 0) return cudaSuccess;
  const int blocks = (int)((n + 255) / 256 < 16384 ? (n + 255) / 256 : 16384);
  scatter_errors_kernel<<<blocks, 256, 0, s>>>(cand, e, n, G, out);
  return cudaGetLastError();
}

cudaError_t launch_refine(const Cand* cand, const float* cand_e, int64_t n, int64_t P, int64_t G, int64_t k,
                          const float* X, const float* b0, float b1, unsigned int* hist, float* Xt, float2* cut,
                          Cand* out, unsigned long long* count, int sms, cudaStream_t s) {
  cudaError_t e = cudaMemsetAsync(hist, 0, sizeof(unsigned int) * (size_t)G * kCandBins, s);
  if (e == cudaSuccess) e = cudaMemsetAsync(count, 0, sizeof(unsigned long long), s);
  if (e != cudaSuccess) return e;
  if (G <= 0) return cudaSuccess;
  const int blocks = (int)((n + 255) / 256 < 16384 ? (n + 255) / 256 : 16384);
  if (n > 0 && G <= kSmemHistGenes) {
    static std::atomic<uint64_t> attr{0};
    e = set_smem_once(attr, cand_hist_smem_kernel, (int)(sizeof(unsigned int) * kCandBins * kSmemHistGenes));
    if (e != cudaSuccess) return e;
    const int hb = (int)((n + 8191) / 8192 < sms ? (n + 8191) / 8192 : sms);
    cand_hist_smem_kernel<<<hb, 1024, sizeof(unsigned int) * kCandBins * (size_t)G, s>>>(cand, cand_e, n, (int)G, b0, b1,
                                                                                        hist);
  } else if (n > 0) {
    cand_hist_kernel<<<blocks, 256, 0, s>>>(cand, cand_e, n, b0, b1, hist);
  }
  refine_kernel<<<(unsigned)G, 256, 0, s>>>(hist, P, G, k, X, b0, b1, Xt, cut);
  if (n > 0) cand_filter_kernel<<<blocks, 256, 0, s>>>(cand, cand_e, n, Xt, cut, out, count);
  return cudaGetLastError();
}


// Surrogate screen of particle p against gene g under the predicted
// statistics (mean mu_pk, predictive std sd_pk), a = sqrt(w_gk):
//   mode 0, per-statistic lower bound
//     L_pg = sum_k max(0, |a (d_gk - mu_pk)| - z a sd_pk)^2 / K;
//   mode 1, lower quantile of the error's predictive distribution: with
//     s_pk ~ N(mu_pk, sd_pk^2) independent, err = sum_k a^2 (d - s)^2 / K has
//     mean m = sum_k (delta^2 + sig^2) / K and variance
//     v = sum_k (2 sig^4 + 4 sig^2 delta^2) / K^2 (delta = a (d - mu),
//     sig = a sd), and L_pg = m - z sqrt(v).
// keep[p] = 1 when L_pg <= X[g] for some gene (X = calibrated threshold).  A
// draw is dropped only when it is confidently far from every gene.  Tiles of
// 128 draws x 128 genes, 8 x 8 per thread, as dist_fast_kernel.
template <int MODE>
__global__ void __launch_bounds__(256) dist_screen_kernel(const float* __restrict__ mu,
                                                          const float* __restrict__ var,
                                                          const float* __restrict__ sw,
                                                          const float* __restrict__ dw, int64_t P, int64_t G,
                                                          int K, const float* __restrict__ X, float z,
                                                          uint8_t* keep, float* err_out) {
  constexpr int GJ = 8, N2 = MODE ? 8 : 1, M2 = MODE ? GJ : 1, kGenes = 16 * GJ;
  __shared__ float sm[kDistKc][kDistTile + 1];
  __shared__ float sv[kDistKc][kDistTile + 1];
  __shared__ float sa[kDistKc][kGenes + 1];
  __shared__ float sd[kDistKc][kGenes + 1];
  const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
  const int64_t g0 = (int64_t)blockIdx.x * kGenes;
  const int64_t p0 = (int64_t)blockIdx.y * kDistTile;
  float acc[8][GJ], acc2[N2][M2];
#pragma unroll
  for (int i = 0; i < 8; ++i)
#pragma unroll
    for (int j = 0; j < GJ; ++j) acc[i][j] = 0.0f;
#pragma unroll
  for (int i = 0; i < N2; ++i)
#pragma unroll
    for (int j = 0; j < M2; ++j) acc2[i][j] = 0.0f;
  for (int k0 = 0; k0 < K; k0 += kDistKc) {
    for (int idx = threadIdx.x; idx < kDistKc * kDistTile; idx += 256) {
      const int r = idx / kDistKc, kk = idx - (idx / kDistKc) * kDistKc;
      const int k = k0 + kk;
      const int64_t p = p0 + r, g = g0 + r;
      float m = 0.0f, v = 0.0f, a = 0.0f, d = 0.0f;
      if (p < P && k < K) {
        m = mu[p * K + k];
        v = sqrtf(fmaxf(var[p * K + k], 0.0f));  // predictive std
        if (MODE == 0) v *= z;
      }
      if (r < kGenes && g < G && k < K) {
        a = sw[g * K + k];
        d = dw[g * K + k];
      }
      sm[kk][r] = m;
      sv[kk][r] = v;
      if (r < kGenes) {
        sa[kk][r] = a;
        sd[kk][r] = d;
      }
    }
    __syncthreads();
    const int kc = (K - k0) < kDistKc ? (K - k0) : kDistKc;
#pragma unroll 2
    for (int kk = 0; kk < kc; ++kk) {
      float m[8], v[8], a[GJ], d[GJ];
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        m[i] = sm[kk][ty + 16 * i];
        v[i] = sv[kk][ty + 16 * i];
      }
#pragma unroll
      for (int j = 0; j < GJ; ++j) {
        a[j] = sa[kk][tx + 16 * j];
        d[j] = sd[kk][tx + 16 * j];
      }
#pragma unroll
      for (int i = 0; i < 8; ++i)
#pragma unroll
        for (int j = 0; j < GJ; ++j) {
          if (MODE == 0) {
            const float t = fmaxf(fabsf(fmaf(-a[j], m[i], d[j])) - a[j] * v[i], 0.0f);
            acc[i][j] = fmaf(t, t, acc[i][j]);
          } else {
            const float dl = fmaf(-a[j], m[i], d[j]);
            const float sg = a[j] * v[i];
            const float s2 = sg * sg, d2 = dl * dl;
            acc[i][j] += d2 + s2;
            acc2[i & (N2 - 1)][j & (M2 - 1)] = fmaf(s2, fmaf(4.0f, d2, 2.0f * s2), acc2[i & (N2 - 1)][j & (M2 - 1)]);
          }
        }
    }
    __syncthreads();
  }
  const float invK = 1.0f / (float)K;
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    const int64_t p = p0 + ty + 16 * i;
    if (p >= P) continue;
    bool any = false;
#pragma unroll
    for (int j = 0; j < GJ; ++j) {
      const int64_t g = g0 + tx + 16 * j;
      if (g >= G) continue;
      // not clipped: far draws keep large predicted errors
      float e = acc[i][j] * invK;
      if (MODE == 1) e -= z * sqrtf(acc2[i & (N2 - 1)][j & (M2 - 1)]) * invK;
      if (err_out) err_out[p * G + g] = e;
      any = any || (e <= X[g]);
    }
    if (any) keep[p] = 1;
  }
}

// The same for up to GC genes: a thread takes a draw, with the errors to every
// gene in registers, and reads the genes' terms of a statistic as broadcasts.
// What bounds it is the shared-memory reads: 2 + GC / 2 words per statistic and
// draw, where the tile of draws x genes reads 2 per gene, padding included (65,536 draws
// x 53 statistics x 4 genes: 108 us in tiles of 128 genes, 32 in tiles of 16,
// 15 here).
constexpr int kScreenRows = 128, kScreenKc = 32;
template <int MODE, int GC>
__global__ void __launch_bounds__(kScreenRows) dist_screen_rows_kernel(const float* __restrict__ mu,
                                                                       const float* __restrict__ var,
                                                                       const float* __restrict__ sw,
                                                                       const float* __restrict__ dw, int64_t P, int G,
                                                                       int K, const float* __restrict__ X, float z,
                                                                       uint8_t* keep, float* err_out) {
  __shared__ float sm[kScreenRows][kScreenKc + 1], sv[kScreenRows][kScreenKc + 1];
  __shared__ float4 sa[kScreenKc][GC / 4], sd[kScreenKc][GC / 4];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int64_t p0 = (int64_t)blockIdx.x * kScreenRows;
  float acc[GC], acc2[MODE ? GC : 1];
#pragma unroll
  for (int j = 0; j < GC; ++j) acc[j] = 0.0f;
#pragma unroll
  for (int j = 0; j < (MODE ? GC : 1); ++j) acc2[j] = 0.0f;
  for (int k0 = 0; k0 < K; k0 += kScreenKc) {
    const int k = k0 + lane;
    // a warp's 32 rows, eight at a time
    for (int r0 = warp * 32; r0 < warp * 32 + 32; r0 += 8) {
      float m[8], v[8];
#pragma unroll
      for (int u = 0; u < 8; ++u) {
        const int64_t p = p0 + r0 + u;
        const bool in = p < P && k < K;
        m[u] = in ? mu[p * K + k] : 0.0f;
        v[u] = in ? var[p * K + k] : 0.0f;
      }
#pragma unroll
      for (int u = 0; u < 8; ++u) {
        const float s = sqrtf(fmaxf(v[u], 0.0f));  // predictive std
        sm[r0 + u][lane] = m[u];
        sv[r0 + u][lane] = MODE == 0 ? s * z : s;
      }
    }
    for (int q = threadIdx.x; q < kScreenKc * GC; q += kScreenRows) {
      const int g = q / kScreenKc, kk = q - g * kScreenKc;
      const bool in = g < G && k0 + kk < K;
      reinterpret_cast<float*>(sa[kk])[g] = in ? sw[(int64_t)g * K + k0 + kk] : 0.0f;
      reinterpret_cast<float*>(sd[kk])[g] = in ? dw[(int64_t)g * K + k0 + kk] : 0.0f;
    }
    __syncthreads();
    const int kc = (K - k0) < kScreenKc ? (K - k0) : kScreenKc;
#pragma unroll 2
    for (int kk = 0; kk < kc; ++kk) {
      const float m = sm[threadIdx.x][kk], v = sv[threadIdx.x][kk];
#pragma unroll
      for (int q = 0; q < GC / 4; ++q) {
        const float4 a4 = sa[kk][q], d4 = sd[kk][q];
        const float a[4] = {a4.x, a4.y, a4.z, a4.w}, d[4] = {d4.x, d4.y, d4.z, d4.w};
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          const int j = 4 * q + u;
          if (MODE == 0) {
            const float t = fmaxf(fabsf(fmaf(-a[u], m, d[u])) - a[u] * v, 0.0f);
            acc[j] = fmaf(t, t, acc[j]);
          } else {
            const float dl = fmaf(-a[u], m, d[u]);
            const float sg = a[u] * v;
            const float s2 = sg * sg, d2 = dl * dl;
            acc[j] += d2 + s2;
            acc2[MODE ? j : 0] = fmaf(s2, fmaf(4.0f, d2, 2.0f * s2), acc2[MODE ? j : 0]);
          }
        }
      }
    }
    __syncthreads();
  }
  const int64_t p = p0 + threadIdx.x;
  if (p >= P) return;
  const float invK = 1.0f / (float)K;
  bool any = false;
#pragma unroll
  for (int j = 0; j < GC; ++j) {
    if (j >= G) break;
    float e = acc[j] * invK;  // not clipped: far draws keep large predicted errors
    if (MODE == 1) e -= z * sqrtf(acc2[MODE ? j : 0]) * invK;
    if (err_out) err_out[p * G + j] = e;
    any = any || (e <= X[j]);
  }
  if (any) keep[p] = 1;
}

// By rows up to 32 genes, where a draw's errors still fit a thread's registers, in 4, 16 or 32
// accumulators; by tiles of 128 genes, padding included, above.  The whole screening of
// 262,144 draws x 53 statistics, mode 0 / 1: by rows 1.18 / 1.18 ms for 4 genes,
// 1.21 / 1.25 for 16, 1.28 / 1.36 for 32; by tiles 1.53 / 1.94 for 33, 1.56 / 2.00 for 128.
template <int MODE>
static void launch_screen(const float* mu, const float* var, const float* sw, const float* dw, int64_t P, int64_t G,
                          int K, const float* X, float z, uint8_t* keep, float* err_out, cudaStream_t s) {
  const unsigned rows = (unsigned)((P + kScreenRows - 1) / kScreenRows);
  if (G <= 4)
    dist_screen_rows_kernel<MODE, 4><<<rows, kScreenRows, 0, s>>>(mu, var, sw, dw, P, (int)G, K, X, z, keep, err_out);
  else if (G <= 16)
    dist_screen_rows_kernel<MODE, 16><<<rows, kScreenRows, 0, s>>>(mu, var, sw, dw, P, (int)G, K, X, z, keep, err_out);
  else if (G <= 32)
    dist_screen_rows_kernel<MODE, 32><<<rows, kScreenRows, 0, s>>>(mu, var, sw, dw, P, (int)G, K, X, z, keep, err_out);
  else
    dist_screen_kernel<MODE><<<dim3((unsigned)((G + kDistTile - 1) / kDistTile),
                                    (unsigned)((P + kDistTile - 1) / kDistTile)), 256, 0, s>>>(mu, var, sw, dw, P, G, K,
                                                                                              X, z, keep, err_out);
}

cudaError_t launch_dist_screen(const float* mu, const float* var, const float* sw, const float* dw, int64_t P,
                               int64_t G, int K, const float* X, float z, int mode, uint8_t* keep, float* err_out,
                               cudaStream_t s) {
  if (P <= 0 || G <= 0) return cudaSuccess;
  if (mode == 1)
    launch_screen<1>(mu, var, sw, dw, P, G, K, X, z, keep, err_out, s);
  else
    launch_screen<0>(mu, var, sw, dw, P, G, K, X, z, keep, err_out, s);
  return cudaGetLastError();
}

}  // namespace abc
