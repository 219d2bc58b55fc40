// distance_fp64.cu — FP64 side of the distance step: weight preparation, the
// exact recheck in the reference's operation order (bit-identical to the
// oracle; built with -fmad=false), the full FP64 error matrix, and the
// per-gene grouping and (err, index) sort of accepted particles
// (scripts/accepted_particles.jl:20-26: findall + sortperm).
#include <algorithm>
#include <atomic>

#include "smem_attr.h"
#include "distance.cuh"
#include "kernels.h"

namespace abc {

// Terms of every (g, k): den = (se^2 + 0.01 d^2) + eps, rden = RN(1/den), and in
// FP32 sw = sqrt(w), dw = sqrt(w) d with w = rden; den and rden may be null.
__global__ void dist_den_kernel(DistInputs in, double* den, double* rden, float* sw, float* dw) {
  const int64_t n = in.G * in.K;
  const double sig2 = 0.1 * 0.1;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
    const double d = in.data[i], e = in.se[i];
    const double eps = (e + d != 0.0) ? 0.0 : 0.0001;
    const double b = (e * e + sig2 * (d * d)) + eps;
    const double w = 1.0 / b;
    if (den) {
      den[i] = b;
      rden[i] = w;
    }
    const double a = sqrt(w);
    sw[i] = (float)a;
    dw[i] = (float)(a * d);
  }
}

cudaError_t launch_dist_den(const DistInputs& in, double* den, double* rden, float* sw, float* dw, cudaStream_t s) {
  const int64_t n = in.G * in.K;
  if (n <= 0) return cudaSuccess;
  int blocks = (int)((n + 63) / 64 < 4096 ? (n + 63) / 64 : 4096);
  dist_den_kernel<<<blocks, 64, 0, s>>>(in, den, rden, sw, dw);
  return cudaGetLastError();
}

__device__ __forceinline__ double den_term(double d, double e) {
  const double sig2 = 0.1 * 0.1;
  const double eps = (e + d != 0.0) ? 0.0 : 0.0001;
  return (e * e + sig2 * (d * d)) + eps;
}

// s32[r][k] = stats[r * stride][k] rounded to float, r < rows; a warp per row
__global__ void __launch_bounds__(256) dist_rows32_kernel(DistInputs in, float* s32, int64_t rows, int64_t stride) {
  const int lane = threadIdx.x & 31;
  for (int64_t r = (int64_t)blockIdx.x * 8 + (threadIdx.x >> 5); r < rows; r += (int64_t)gridDim.x * 8) {
    const double* src = in.stats + r * stride * in.K;
    for (int k = lane; k < in.K; k += 32) s32[r * in.K + k] = rn32_bits(src[k]);
  }
}

cudaError_t launch_dist_rows32(const DistInputs& in, float* s32, int64_t rows, int64_t stride, cudaStream_t s) {
  if (rows <= 0 || in.K <= 0) return cudaSuccess;
  const int64_t blocks = (rows + 7) / 8;
  dist_rows32_kernel<<<(unsigned)(blocks < 65536 ? blocks : 65536), 256, 0, s>>>(in, s32, rows, stride);
  return cudaGetLastError();
}

// err of one (p, g) pair exactly as compute_trunc_errors / nlsqerror_part
// (scripts/compute_errors.jl:30-43): per family, sum of diff^2 / den in
// order, then part / K added to the total; clipped at 10.
__device__ __forceinline__ double err_exact(const DistInputs& in, int64_t p, int64_t g) {
  const double* s = in.stats + p * in.K;
  const double* d = in.data + g * in.K;
  const double* e = in.se + g * in.K;
  const double nK = (double)in.K;
  double tot = 0.0;
  int k = 0;
  if (in.den) {
    const double* dn = in.den + g * in.K;
    const double* ry = in.rden + g * in.K;
    const double rK = 1.0 / nK;
    for (int f = 0; f < in.n_fam; ++f) {
      double part = 0.0;
      // unrolled for the loads of the next terms beside the chain of additions
#pragma unroll 4
      for (int q = 0; q < in.fam[f]; ++q) {
        const double diff = __ldg(d + k + q) - __ldg(s + k + q);
        part = part + div_rn(diff * diff, __ldg(dn + k + q), __ldg(ry + k + q));
      }
      k += in.fam[f];
      tot = tot + div_rn(part, nK, rK);
    }
  } else {
    for (int f = 0; f < in.n_fam; ++f) {
      double part = 0.0;
      for (int q = 0; q < in.fam[f]; ++q, ++k) {
        const double diff = d[k] - s[k];
        part = part + (diff * diff) / den_term(d[k], e[k]);
      }
      tot = tot + part / nK;
    }
  }
  if (tot > 10.0) tot = 10.0;
  return tot;
}

// FP64 errors of candidates already grouped by gene (sp, sg: particle and gene
// of each entry).  A warp takes 32 consecutive entries and walks the
// statistics in chunks of kRecheckCols columns: it copies the chunk of its 32
// rows into shared memory with coalesced loads (consecutive lanes read
// consecutive values, rows back to back), then each lane adds its pair's terms
// of that chunk from shared memory, carrying the family sums across chunks.
// The gene rows it reads (data, den, rden) are mostly the same for the whole
// warp and are broadcast.  Row stride kRecheckCols + 1 (odd) keeps the lanes'
// column reads on distinct banks; the small chunk keeps 32 warps resident per
// SM, enough to keep the FP64 pipe (the bound: six FP64 operations per term)
// busy.
constexpr int kRecheckWarps = 8;
constexpr int kRecheckCols = 24;
constexpr int kRecheckLd = kRecheckCols + 1;

// WARPS: kRecheckWarps, or 1 while the chunks do not fill the GPU: a term's six
// FP64 operations hold a scheduler's pipe whatever the number of pairs, so
// the warps of a few chunks go to different ones (800 pairs of 53 statistics: 39 us in
// blocks of 8 warps, 30 apart).
template <int WARPS>
__global__ void __launch_bounds__(WARPS * 32) recheck_grouped_kernel(DistInputs in, const int32_t* sp,
                                                                     const int32_t* sg, int64_t n, double* se64) {
  __shared__ double rs_smem[WARPS * 32 * kRecheckLd];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int K = in.K;
  double* S = rs_smem + warp * 32 * kRecheckLd;
  const double nK = (double)K;
  const double rK = 1.0 / nK;
  const int64_t n_chunks = (n + 31) >> 5;
  const int64_t wstride = (int64_t)gridDim.x * WARPS;
  for (int64_t ch = (int64_t)blockIdx.x * WARPS + warp; ch < n_chunks; ch += wstride) {
    const int64_t i = ch * 32 + lane;
    const bool mine = i < n;
    const int32_t p = mine ? sp[i] : 0;
    const int64_t g = mine ? sg[i] : 0;
    const int rows = (int)(n - ch * 32 < 32 ? n - ch * 32 : 32);
    const double* d = in.data + g * K;
    const double* dn = in.den + g * K;
    const double* ry = in.rden + g * K;
    double tot = 0.0, part = 0.0;
    // families: f is the open one, fend the column after its last term
    int f = 0, fend = in.fam[0];
    while (fend == 0 && f < in.n_fam) {  // leading empty families add 0 / K
      tot = tot + div_rn(part, nK, rK);
      ++f;
      fend = f < in.n_fam ? fend + in.fam[f] : -1;
    }
    for (int c0 = 0; c0 < K; c0 += kRecheckCols) {
      const int cw = K - c0 < kRecheckCols ? K - c0 : kRecheckCols;
      // flat copy of rows x cw values: lane takes e = lane + 32 t, (r, c) = divmod(e, cw)
      const int T = (rows * cw + 31) >> 5;
      int r = lane / cw, c = lane - (lane / cw) * cw;
      for (int t0 = 0; t0 < T; t0 += 8) {
        double v[8];
        int dst[8];
#pragma unroll
        for (int u = 0; u < 8; ++u) {
          const int32_t pr = __shfl_sync(0xffffffffu, p, r < 31 ? r : 31);
          const bool take = t0 + u < T && r < rows;
          dst[u] = take ? r * kRecheckLd + c : -1;
          v[u] = take ? __ldg(in.stats + (int64_t)pr * K + c0 + c) : 0.0;
          c += 32;
          while (c >= cw) {
            c -= cw;
            ++r;
          }
        }
#pragma unroll
        for (int u = 0; u < 8; ++u)
          if (dst[u] >= 0) S[dst[u]] = v[u];
      }
      __syncwarp();
      if (mine) {
        const double* s = S + lane * kRecheckLd - c0;
        for (int k = c0; k < c0 + cw;) {
          const int ke = fend > k && fend < c0 + cw ? fend : c0 + cw;  // the open family's terms of this chunk
#pragma unroll 4
          for (; k < ke; ++k) {
            const double diff = __ldg(d + k) - s[k];
            part = part + div_rn(diff * diff, __ldg(dn + k), __ldg(ry + k));
          }
          while (k == fend) {  // close this family and any empty ones after it
            tot = tot + div_rn(part, nK, rK);
            part = 0.0;
            ++f;
            fend = f < in.n_fam ? fend + in.fam[f] : -1;
          }
        }
      }
      __syncwarp();
    }
    if (mine) {
      if (tot > 10.0) tot = 10.0;
      se64[i] = tot;
    }
  }
}

// ---------------------------------------------------------------------------
// Certified FP32 errors for selections that return indices only
// ---------------------------------------------------------------------------
// A candidate's error is evaluated in FP32 from two-float splits of its FP64
// inputs: x = h + l with |x - h - l| <= 2^-47 |x|, |l| <= 2^-23 |x| (data: h =
// RN32(x), l = RN32(x - h); statistics: h = the top 24 significand bits,
// exact integer bit manipulation, l = the remaining 29 bits rounded to float).
// With r = 1/den rounded to float, u = 2^-24:
//   delta = RN(RN(dh - sh) + RN(dl - sl))       (the hi parts cancel exactly)
//   T     = RN(delta RN(delta r))               per statistic
//   S     = Kahan sum of the T, e = RN(S RN(1/K))
// and, writing T* = (d - s)^2 / den for the exact term and a = den^-1/2 (so
// a |d| <= 10 because den >= 0.01 d^2): |delta - (d - s)| <= 2.0001 u |d - s| +
// 2^-45.4 (|d| + |s|), hence |T - T*| <= 7.03 u T* + 2^-44.4 (20 sqrt(T*) + T*)
// + 2^-90 (20 + sqrt(T*))^2; Kahan summation adds <= 2.1 u sum T, the final
// scaling 2.01 u, and the reference's FP64 evaluation differs from the exact
// value by < 1e-14 relative.  Altogether |e - err64| <= 11.2 u err +
// 2^-40 sqrt(err) + 2^-80; 1e-6 e + 1.5e-12 sqrt(e + 1e-12) covers that with a
// 1.5x margin, and approx_bound uses its linear majorant (1e-6 + 1e-12) e +
// 1e-12 (sqrt(x) <= (1 + x) / 2), one FMA instead of an FP64 square root;
// v - B(v) and v + B(v) are increasing in v.  The derivation
// needs every |d|, |s| in {0} u [2^-60, 2^60] (no underflow in the splits),
// den in [2^-120, 2^120] (1/den a normal float; an underflow in delta r then
// costs at most 2^-88 per term, far inside the bound's absolute part) and a
// finite result; other pairs are computed in FP64.
__device__ __forceinline__ bool key_less(double ea, int32_t pa, double eb, int32_t pb);
__device__ __forceinline__ double approx_bound(double v) { return fma(1.000001e-6, v, 1e-12); }

// x = h + l by truncation of the significand, on the two 32-bit halves of x
// (integer operations only): h keeps the sign, the exponent rebiased from 1023
// to 127 and the top 23 stored significand bits; l is the remaining 29 bits
// rounded to float and scaled by 2^(e - 1075).
__device__ __forceinline__ bool split_trunc(double x, float& h, float& l) {
  const unsigned hi = (unsigned)__double2hiint(x), lo = (unsigned)__double2loint(x);
  const unsigned mag = hi & 0x7fffffffu, sign = hi & 0x80000000u;
  const unsigned e = mag >> 20;
  const bool zero = (mag | lo) == 0u;
  const bool ok = zero || e - (1023u - 60u) <= 120u;  // exponent in [-60, 60]
  // ((e - 896) << 23) | (top 20 bits << 3) | (next 3 bits): the float's exponent and significand
  h = __uint_as_float(zero ? 0u : (sign | ((mag - (896u << 20)) << 3) | (lo >> 29)));
  const float r = __uint2float_rn(lo & 0x1fffffffu);
  const float scale = __uint_as_float(((e - 948u) & 0xffu) << 23);  // 2^(e - 1075); garbage when !ok
  l = zero ? 0.0f : __uint_as_float(__float_as_uint(__fmul_rn(r, scale)) | sign);
  return ok;
}

// per (gene, statistic): (h, l, 1/den, 0) with d = h + l
__global__ void ff_prep_genes_kernel(DistInputs in, float4* gt) {
  const int64_t n = in.G * in.K;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
    const double d = in.data[i], den = in.den[i];
    const double ad = fabs(d);
    const bool ok = (d == 0.0 || (ad >= 0x1p-60 && ad <= 0x1p60)) && den >= 0x1p-120 && den <= 0x1p120;
    const float h = (float)d;
    gt[i] = make_float4(h, (float)(d - (double)h), ok ? (float)in.rden[i] : __int_as_float(0x7fc00000), 0.0f);
  }
}

// Candidates grouped by gene, statistics rows staged as in
// recheck_grouped_kernel.  v[i] = the certified FP32 error (10 exactly when
// it lies above 10 by more than its bound); pairs outside the derivation's
// range get their position appended to pos (FP64 later).
// Blocks of four warps: a warp's share of shared memory is free again sooner (2.01 ms
// for 10.9 million pairs of 72 statistics, 2.13 in blocks of eight).
constexpr int kApproxWarps = 4;
__global__ void __launch_bounds__(kApproxWarps * 32) approx_grouped_kernel(DistInputs in, const int32_t* sp,
                                                                            const int32_t* sg, int64_t n,
                                                                            const float4* gt, float rK, double* v,
                                                                            int32_t* pos,
                                                                            unsigned long long* count) {
  __shared__ double rs_smem[kApproxWarps * 32 * kRecheckLd];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int K = in.K;
  double* S = rs_smem + warp * 32 * kRecheckLd;
  const int64_t n_chunks = (n + 31) >> 5;
  const int64_t wstride = (int64_t)gridDim.x * kApproxWarps;
  for (int64_t ch = (int64_t)blockIdx.x * kApproxWarps + warp; ch < n_chunks; ch += wstride) {
    const int64_t i = ch * 32 + lane;
    const bool mine = i < n;
    const int32_t p = mine ? sp[i] : 0;
    const int64_t g = mine ? sg[i] : 0;
    const int rows = (int)(n - ch * 32 < 32 ? n - ch * 32 : 32);
    const float4* gk = gt + g * K;
    float acc = 0.0f, comp = 0.0f;
    bool ok = true;
    for (int c0 = 0; c0 < K; c0 += kRecheckCols) {
      const int cw = K - c0 < kRecheckCols ? K - c0 : kRecheckCols;
      const int T = (rows * cw + 31) >> 5;
      int r = lane / cw, c = lane - (lane / cw) * cw;
      for (int t0 = 0; t0 < T; t0 += 8) {
        double vv[8];
        int dst[8];
#pragma unroll
        for (int u = 0; u < 8; ++u) {
          const int32_t pr = __shfl_sync(0xffffffffu, p, r < 31 ? r : 31);
          const bool take = t0 + u < T && r < rows;
          dst[u] = take ? r * kRecheckLd + c : -1;
          vv[u] = take ? __ldg(in.stats + (int64_t)pr * K + c0 + c) : 0.0;
          c += 32;
          while (c >= cw) {
            c -= cw;
            ++r;
          }
        }
#pragma unroll
        for (int u = 0; u < 8; ++u)
          if (dst[u] >= 0) S[dst[u]] = vv[u];
      }
      __syncwarp();
      if (mine) {
        const double* s = S + lane * kRecheckLd - c0;
        for (int k = c0; k < c0 + cw; ++k) {
          float sh, sl;
          ok = split_trunc(s[k], sh, sl) && ok;
          const float4 q = __ldg(gk + k);
          const float x = __fsub_rn(q.x, sh);
          const float y = __fsub_rn(q.y, sl);
          const float dd = __fadd_rn(x, y);
          const float term = __fmul_rn(dd, __fmul_rn(dd, q.z));
          const float yk = __fsub_rn(term, comp);
          const float t = __fadd_rn(acc, yk);
          comp = __fsub_rn(__fsub_rn(t, acc), yk);
          acc = t;
        }
      }
      __syncwarp();
    }
    if (mine) {
      const float e = __fmul_rn(acc, rK);
      ok = ok && e == e && e < INFINITY;
      if (ok) {
        const double ed = (double)e;
        v[i] = ed - approx_bound(ed) >= 10.0 ? 10.0 : ed;
      } else {
        v[i] = 0.0;
        pos[atomicAdd(count, 1ull)] = (int32_t)i;
      }
    }
  }
}

// E[pos[j]] = the FP64 error of the pair at that position, j < *count
__global__ void recheck_list_kernel(DistInputs in, const int32_t* sp, const int32_t* sg, const int32_t* pos,
                                    const unsigned long long* count, double* E) {
  const int64_t m = (int64_t)*count;
  for (int64_t j = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; j < m; j += (int64_t)gridDim.x * blockDim.x) {
    const int32_t i = pos[j];
    E[i] = err_exact(in, sp[i], sg[i]);
  }
}

// After the sort by the certified values: a position whose interval
// [v - B(v), v + B(v)] overlaps a neighbour's in its gene's list, or holds
// the clip value 10 or the gene's threshold (modes 0 and 2), is appended to pos
// and its gene marked dirty.  Intervals have increasing ends along the sorted
// list, so an interval that overlaps no neighbour overlaps no other; every
// other pair is then in its exact place, and exact values for the listed
// pairs plus one more sort give the exact order.
__global__ void ambiguous_kernel(const int32_t* sg, const int64_t* goff, const double* E, int64_t n, int mode,
                                 double eps_all, const double* eps_g, int32_t* pos, unsigned long long* count,
                                 uint8_t* flag) {
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
    const double v = E[i];
    if (v != v) continue;  // NaN: exact (FP64 path), sorts last
    const int64_t g = sg[i];
    const int64_t a = goff[g], b = goff[g + 1];
    const double B = approx_bound(v);
    bool amb = fabs(v - 10.0) <= B;
    if (i > a) {
      const double w = E[i - 1];
      if (w == w && w + approx_bound(w) >= v - B) amb = true;
    }
    if (i + 1 < b) {
      const double w = E[i + 1];
      if (w == w && v + B >= w - approx_bound(w)) amb = true;
    }
    if (mode != 1) {
      const double thr = eps_g ? eps_g[g] : eps_all;
      if (fabs(v - thr) <= B) amb = true;
    }
    flag[i] = amb ? 1 : 0;
    if (amb) pos[atomicAdd(count, 1ull)] = (int32_t)i;
  }
}

// After the FP64 values of the flagged positions are in: every maximal run
// of consecutive flagged positions in a gene's list is sorted in place by
// (err, p) (the neighbours of a run have intervals wholly below or above it,
// so nothing else moves); a run longer than kRunSort marks its gene for a
// full re-sort instead.
constexpr int kRunSort = 64;

__global__ void run_sort_kernel(const int32_t* sg, const int64_t* goff, const uint8_t* flag, int64_t n,
                                int32_t* sp, double* E, int* dirty) {
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
    if (!flag[i]) continue;
    const int64_t g = sg[i];
    const int64_t a = goff[g], b = goff[g + 1];
    if (i > a && flag[i - 1]) continue;  // not the start of a run
    int64_t e = i + 1;
    while (e < b && flag[e] && e - i <= kRunSort) ++e;
    if (e - i > kRunSort) {
      dirty[g] = 1;
      continue;
    }
    for (int64_t j = i + 1; j < e; ++j) {  // insertion sort
      const double x = E[j];
      const int32_t px = sp[j];
      int64_t k = j - 1;
      while (k >= i && key_less(x, px, E[k], sp[k])) {
        E[k + 1] = E[k];
        sp[k + 1] = sp[k];
        --k;
      }
      E[k + 1] = x;
      sp[k + 1] = px;
    }
  }
}

// Full error matrix.  Errors are clipped at 10, and of a matrix over prior
// draws most are: a block first evaluates its ROWS x cols pairs in
// FP32 (two FMAs per term, as dist_fast_kernel) and writes 10 where that is
// certain; only the other pairs are computed in FP64, whose narrow pipe took
// the whole 0.97 ms for 3,001 x 500 pairs of 53 statistics (0.08 with 0.4 %
// of them below the clip; with all of them below it, as before).  Particles and
// genes per block: launch_dist_full.
// Certain: K e32 > K sure.  With finite operands |e32 - e| <= B(e) =
// 1.5 u (64 sqrt(e) + (K + 8) e) (distance.cuh), so e <= 10 implies e32 <= 10 + B(10), and
// sure is 10 + 2 B(10).  An operand that is not finite in FP32 becomes
// NaN, which no comparison holds for, so its pairs are computed in FP64.
constexpr int kFullRows = 32, kFullTile = 64, kFullKc = 16;  // particles and genes at most, statistics
__device__ __forceinline__ float finite_or_nan(float x) { return fabsf(x) < INFINITY ? x : __int_as_float(0x7fc00000); }

template <int ROWS>
__global__ void __launch_bounds__(256) dist_full_kernel(DistInputs in, const float* __restrict__ sw,
                                                        const float* __restrict__ dw, float sure, int even, double* err) {
  const int cols = ROWS == kFullRows ? kFullTile : even;  // genes per tile
  // threads: TY particles x TX genes, RI x GJ pairs each
  constexpr int TY = ROWS < 16 ? ROWS : 16, TX = 256 / TY, RI = ROWS / TY, GJ = kFullTile / TX;
  static_assert(ROWS <= kFullTile && TX <= kFullTile, "the tile's pairs fall to 256 threads");
  __shared__ float ss[kFullKc][ROWS + 1], sa[kFullKc][kFullTile + 1], sd[kFullKc][kFullTile + 1];
  __shared__ unsigned short todo[ROWS * kFullTile];
  __shared__ int n_todo;
  const int tx = threadIdx.x % TX, ty = threadIdx.x / TX, lane = threadIdx.x & 31;
  const int64_t g0 = (int64_t)blockIdx.x * cols;
  if (threadIdx.x == 0) n_todo = 0;
  for (int64_t p0 = (int64_t)blockIdx.y * ROWS; p0 < in.P; p0 += (int64_t)gridDim.y * ROWS) {
    float acc[RI][GJ];
#pragma unroll
    for (int i = 0; i < RI; ++i)
#pragma unroll
      for (int j = 0; j < GJ; ++j) acc[i][j] = 0.0f;
    for (int k0 = 0; k0 < in.K; k0 += kFullKc) {
      __syncthreads();
      for (int q = threadIdx.x; q < kFullKc * kFullTile; q += 256) {
        const int r = q / kFullKc, kk = q - r * kFullKc, k = k0 + kk;
        const int64_t p = p0 + r, g = g0 + r;
        float s = 0.0f, a = 0.0f, d = 0.0f;
        if (k < in.K) {
          if (r < ROWS && p < in.P) s = finite_or_nan(rn32_bits(in.stats[p * in.K + k]));
          if (g < in.G) {
            a = finite_or_nan(sw[g * in.K + k]);
            d = finite_or_nan(dw[g * in.K + k]);
          }
        }
        if (r < ROWS) ss[kk][r] = s;
        sa[kk][r] = a;
        sd[kk][r] = d;
      }
      __syncthreads();
#pragma unroll 4
      for (int kk = 0; kk < kFullKc; ++kk) {
        float s[RI], a[GJ], d[GJ];
#pragma unroll
        for (int i = 0; i < RI; ++i) s[i] = ss[kk][ty + TY * i];
#pragma unroll
        for (int j = 0; j < GJ; ++j) {
          a[j] = sa[kk][tx + TX * j];
          d[j] = sd[kk][tx + TX * j];
        }
#pragma unroll
        for (int i = 0; i < RI; ++i)
#pragma unroll
          for (int j = 0; j < GJ; ++j) {
            const float t = fmaf(-a[j], s[i], d[j]);
            acc[i][j] = fmaf(t, t, acc[i][j]);
          }
      }
    }
    const float limit = sure * (float)in.K;
#pragma unroll
    for (int i = 0; i < RI; ++i)
#pragma unroll
      for (int j = 0; j < GJ; ++j) {
        const int r = ty + TY * i, c = tx + TX * j;
        const bool real = p0 + r < in.P && c < cols && g0 + c < in.G;
        const bool clip = acc[i][j] > limit;
        if (real && clip) err[(p0 + r) * in.G + g0 + c] = 10.0;
        const unsigned m = __ballot_sync(0xffffffffu, real && !clip);
        int base = 0;
        if (lane == 0 && m) base = atomicAdd(&n_todo, __popc(m));
        base = __shfl_sync(0xffffffffu, base, 0);
        if (real && !clip) todo[base + __popc(m & ((1u << lane) - 1u))] = (unsigned short)(r * kFullTile + c);
      }
    __syncthreads();
    const int n = n_todo;
    for (int q = threadIdx.x; q < n; q += 256) {
      const int64_t p = p0 + todo[q] / kFullTile, g = g0 + todo[q] % kFullTile;
      err[p * in.G + g] = err_exact(in, p, g);
    }
    __syncthreads();
    if (threadIdx.x == 0) n_todo = 0;
  }
}

template <int ROWS>
static cudaError_t launch_full(const DistInputs& in, const float* sw, const float* dw, int64_t tiles, double* err,
                               cudaStream_t s) {
  const float sure = 10.0f + 2.0f * dist_bound_f(10.0f, in.K);
  const int64_t py = (in.P + ROWS - 1) / ROWS;
  dim3 grid((unsigned)tiles, (unsigned)(py < 65535 ? py : 65535));
  dist_full_kernel<ROWS><<<grid, 256, 0, s>>>(in, sw, dw, sure, (int)((in.G + tiles - 1) / tiles), err);
  return cudaGetLastError();
}

// 32 particles per tile read the genes' terms least often, but where few pairs are
// clipped a thread computes eight of them one after the other, and with few blocks that
// chain is the call: the most particles are taken for which every multiprocessor still
// gets two blocks, and below 32 the genes are split evenly over the tiles.
// Milliseconds of the whole call, 53 statistics, few pairs below the clip / all:
//                a thread per pair   32 particles    by this rule
//   64 x 64         0.088 / 0.088    0.055 / 0.277   0.045 / 0.080
//   500 x 50        0.092 / 0.091    0.057 / 0.241   0.057 / 0.081
//   700 x 100       0.120 / 0.120    0.073 / 0.308   0.073 / 0.134
//   500 x 300       0.193 / 0.192    0.083 / 0.318   0.084 / 0.211
//   200 x 2,000     0.561 / 0.562    0.114 / 0.483   0.112 / 0.387
//   2,000 x 300     0.714 / 0.715    0.111 / 0.659   32 particles
cudaError_t launch_dist_full(const DistInputs& in, const float* sw, const float* dw, double* err, cudaStream_t s) {
  if (in.P <= 0 || in.G <= 0) return cudaSuccess;
  const int64_t tiles = (in.G + kFullTile - 1) / kFullTile;
  auto fills = [&](int rows) { return (in.P + rows - 1) / rows * tiles >= 2 * (int64_t)in.sms; };
  if (fills(kFullRows)) return launch_full<kFullRows>(in, sw, dw, tiles, err, s);
  if (fills(16)) return launch_full<16>(in, sw, dw, tiles, err, s);
  if (fills(8)) return launch_full<8>(in, sw, dw, tiles, err, s);
  return launch_full<4>(in, sw, dw, tiles, err, s);
}

// ---------------------------------------------------------------------------
// grouping by gene: count, exclusive scan, scatter
// ---------------------------------------------------------------------------
__global__ void gene_count_kernel(const Cand* cand, int64_t n, int64_t* gcount) {
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
    atomicAdd((unsigned long long*)&gcount[cand[i].g], 1ull);
}

// The same count with a per-block histogram in shared memory (G counters):
// one global atomic per (block, gene) instead of one per candidate, which
// all land on a few thousand addresses.
__global__ void __launch_bounds__(256) gene_count_smem_kernel(const Cand* cand, int64_t n, int G, int64_t chunk,
                                                              int64_t* gcount) {
  extern __shared__ unsigned int h[];
  for (int g = threadIdx.x; g < G; g += blockDim.x) h[g] = 0u;
  __syncthreads();
  const int64_t b0 = (int64_t)blockIdx.x * chunk, b1 = b0 + chunk < n ? b0 + chunk : n;
  for (int64_t i = b0 + threadIdx.x; i < b1; i += blockDim.x) atomicAdd(&h[cand[i].g], 1u);
  __syncthreads();
  for (int g = threadIdx.x; g < G; g += blockDim.x)
    if (h[g]) atomicAdd((unsigned long long*)&gcount[g], (unsigned long long)h[g]);
}

// Scatter of a contiguous chunk per block: local counts per gene, one global
// reservation per (block, gene), then positions from shared-memory atomics.
__global__ void __launch_bounds__(256) scatter_smem_kernel(const Cand* cand, int64_t n, int G, int64_t chunk,
                                                           const int64_t* goff, unsigned long long* cursor,
                                                           int32_t* sp, int32_t* sg) {
  extern __shared__ unsigned long long sb[];  // G reserved bases, then G local counters
  unsigned int* cnt = reinterpret_cast<unsigned int*>(sb + G);
  for (int g = threadIdx.x; g < G; g += blockDim.x) cnt[g] = 0u;
  __syncthreads();
  const int64_t b0 = (int64_t)blockIdx.x * chunk, b1 = b0 + chunk < n ? b0 + chunk : n;
  for (int64_t i = b0 + threadIdx.x; i < b1; i += blockDim.x) atomicAdd(&cnt[cand[i].g], 1u);
  __syncthreads();
  for (int g = threadIdx.x; g < G; g += blockDim.x) {
    const unsigned int c = cnt[g];
    sb[g] = c ? (unsigned long long)goff[g] + atomicAdd(&cursor[g], (unsigned long long)c) : 0ull;
    cnt[g] = 0u;
  }
  __syncthreads();
  for (int64_t i = b0 + threadIdx.x; i < b1; i += blockDim.x) {
    const Cand c = cand[i];
    const unsigned long long pos = sb[c.g] + atomicAdd(&cnt[c.g], 1u);
    sp[pos] = c.p;
    sg[pos] = c.g;
  }
}

__global__ void __launch_bounds__(1024) scan_kernel(const int64_t* cnt, int64_t G, int64_t* off) {
  __shared__ int64_t wsum[32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int64_t per = (G + 1023) / 1024;
  const int64_t b = threadIdx.x * per;
  int64_t own = 0;
  for (int64_t i = b; i < b + per && i < G; ++i) own += cnt[i];
  int64_t run = own;  // inclusive scan over the warp, then over the warps
  for (int o = 1; o < 32; o <<= 1) {
    const int64_t v = __shfl_up_sync(0xffffffffu, run, o);
    if (lane >= o) run += v;
  }
  if (lane == 31) wsum[warp] = run;
  __syncthreads();
  if (warp == 0) {
    int64_t w = wsum[lane];
    for (int o = 1; o < 32; o <<= 1) {
      const int64_t v = __shfl_up_sync(0xffffffffu, w, o);
      if (lane >= o) w += v;
    }
    wsum[lane] = w;
  }
  __syncthreads();
  run += (warp ? wsum[warp - 1] : 0) - own;
  for (int64_t i = b; i < b + per && i < G; ++i) {
    off[i] = run;
    run += cnt[i];
  }
  if (b + per >= G && b < G) off[G] = run;
  if (G == 0 && threadIdx.x == 0) off[0] = 0;
}

__global__ void scatter_kernel(const Cand* cand, int64_t n, const int64_t* goff, unsigned long long* cursor,
                               int32_t* sp, int32_t* sg) {
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
    Cand c = cand[i];
    unsigned long long pos = (unsigned long long)goff[c.g] + atomicAdd(&cursor[c.g], 1ull);
    sp[pos] = c.p;
    sg[pos] = c.g;
  }
}

// Per-gene sort by (err, p), NaN last, ties by index, a block per gene, on keys
// that are the bit patterns of the errors (monotone for the non-negative
// errors; NaN canonicalised to one pattern).
// - up to kSortDirect entries: each thread counts the entries below its own;
// - longer lists: entries go to 4,096 bins, a monotone map of (error, index):
//   3,072 equal bins of the range of the errors below the clip value in FP32, then
//   1,023 equal ranges of the particle index for errors at the clip value, where ties
//   are the rule, then everything above.  Up to kSortCap entries in shared
//   memory, longer lists by way of tmp_key and tmp_p (as many entries as the list).
//   Windows of whole bins are then finished in shared memory: each entry
//   counts those below it in its bin, or, where a bin holds more than kBinMax,
//   the window goes through a bitonic network;
// - a bin of more than kSortCap entries (ties elsewhere than at the clip value):
//   a bitonic network over the list in global memory.
// Bound by latency of shared memory and barriers; two blocks of 512 threads per
// SM (112 KB each) overlap them.  2,000 lists of 5,450 entries take 0.234 ms (a
// bitonic network over 8,192 register entries: 1.69).
__device__ __forceinline__ bool key_less(double ea, int32_t pa, double eb, int32_t pb) {
  const bool na = ea != ea, nb = eb != eb;
  if (na != nb) return nb;
  if (na) return pa < pb;
  return ea < eb || (ea == eb && pa < pb);
}

constexpr uint64_t kNanKey = 0x7ff8000000000000ull;

__device__ __forceinline__ uint64_t err_key(double e) {
  if (e != e) return kNanKey;
  if (e == 0.0) return 0ull;  // +0 and -0
  return (uint64_t)__double_as_longlong(e);
}

__device__ __forceinline__ bool sort_key_less(uint64_t ka, int32_t pa, uint64_t kb, int32_t pb) {
  return ka < kb || (ka == kb && pa < pb);
}
__device__ __forceinline__ bool sort_key_less(double ea, int32_t pa, double eb, int32_t pb) {
  return key_less(ea, pa, eb, pb);
}

constexpr int kSortThreads = 512, kSortCap = 8192, kSortBins = 4096, kSortDirect = 256, kBinMax = 512;
constexpr int kValueBins = 3072;
constexpr uint64_t kClipKey = 0x4024000000000000ull;  // 10.0
constexpr int kSortSmem = kSortCap * (int)(sizeof(uint64_t) + sizeof(int32_t)) + kSortBins * (int)sizeof(int);

// FP32 value of a key that is not NaN; rounding to nearest keeps the order
__device__ __forceinline__ float key_value(uint64_t key) { return rn32_bits(__longlong_as_double((long long)key)); }

// The map to bins.  Non-decreasing in (key, p): every step rounds monotonically.
// A range of zero width (scale 0 or infinite) sends all of it to one bin.
struct SortMap {
  float lo, scale, p_scale;
  int p_lo;
  __device__ __forceinline__ int bin(uint64_t key, int32_t p) const {
    if (key < kClipKey) return (int)fminf((key_value(key) - lo) * scale, (float)(kValueBins - 1));
    if (key > kClipKey) return kSortBins - 1;
    return kValueBins + (int)fminf((float)(p - p_lo) * p_scale, (float)(kSortBins - kValueBins - 2));
  }
};

// All-ascending bitonic network (the first step of every merge of size k pairs
// i with i ^ (k - 1), the others i with i ^ j) over n2, a power of two, entries
// of K and P; those from n on are absent and above all others.
template <typename Key>
__device__ void bitonic(Key* K, int32_t* P, int64_t n, int64_t n2) {
  for (int64_t k = 2; k <= n2; k <<= 1) {
    for (int64_t j = k >> 1; j > 0; j >>= 1) {
      const int64_t flip = j == (k >> 1) ? k - 1 : j;
      for (int64_t i = threadIdx.x; i < n; i += kSortThreads) {
        const int64_t q = i ^ flip;
        if (q > i && q < n) {
          const Key ka = K[i], kb = K[q];
          const int32_t pa = P[i], pb = P[q];
          if (sort_key_less(kb, pb, ka, pa)) {
            K[i] = kb;
            K[q] = ka;
            P[i] = pb;
            P[q] = pa;
          }
        }
      }
      __syncthreads();
    }
  }
}

__global__ void __launch_bounds__(kSortThreads, 2) segsort_kernel(const int64_t* goff, int32_t* sp, double* se64,
                                                                  const int* dirty, uint64_t* tmp_key,
                                                                  int32_t* tmp_p) {
  extern __shared__ uint64_t sort_smem[];
  __shared__ unsigned int s_lo, s_hi, s_plo, s_phi;
  __shared__ int s_warp[kSortThreads / 32], s_most;
  const int64_t g = blockIdx.x;
  if (dirty && !dirty[g]) return;
  const int64_t base = goff[g];
  const int64_t n = goff[g + 1] - base;
  if (n <= 1) return;
  const int t = threadIdx.x, lane = t & 31;
  int32_t* P = sp + base;
  double* E = se64 + base;
  uint64_t* sK = sort_smem;
  int32_t* sP = reinterpret_cast<int32_t*>(sK + kSortCap);
  int* bins = sP + kSortCap;
  if (n <= kSortDirect) {
    const int m = (int)n;
    uint64_t key = 0;
    int32_t p = 0;
    if (t < m) {
      sK[t] = key = err_key(E[t]);
      sP[t] = p = P[t];
    }
    __syncthreads();
    if (t < m) {
      int r = 0;
#pragma unroll 4
      for (int j = 0; j < m; ++j) r += sort_key_less(sK[j], sP[j], key, p) ? 1 : 0;
      E[r] = __longlong_as_double((long long)key);
      P[r] = p;
    }
    return;
  }
  // range of the errors below the clip value, as FP32 (the patterns of
  // non-negative floats are ordered), and of the indices at it
  if (t == 0) {
    s_lo = s_plo = 0xffffffffu;
    s_hi = s_phi = 0;
    s_most = 0;
  }
  for (int b = t; b < kSortBins; b += kSortThreads) bins[b] = 0;
  __syncthreads();
  unsigned int lo_u = 0xffffffffu, hi_u = 0, plo_u = 0xffffffffu, phi_u = 0;
#pragma unroll 4
  for (int64_t i = t; i < n; i += kSortThreads) {
    const uint64_t key = err_key(E[i]);
    const unsigned int p = (unsigned int)P[i];
    if (key < kClipKey) {
      const unsigned int u = __float_as_uint(key_value(key));
      lo_u = min(lo_u, u);
      hi_u = max(hi_u, u);
    } else if (key == kClipKey) {
      plo_u = min(plo_u, p);
      phi_u = max(phi_u, p);
    }
  }
  lo_u = __reduce_min_sync(0xffffffffu, lo_u);
  hi_u = __reduce_max_sync(0xffffffffu, hi_u);
  plo_u = __reduce_min_sync(0xffffffffu, plo_u);
  phi_u = __reduce_max_sync(0xffffffffu, phi_u);
  if (lane == 0) {
    atomicMin(&s_lo, lo_u);
    atomicMax(&s_hi, hi_u);
    atomicMin(&s_plo, plo_u);
    atomicMax(&s_phi, phi_u);
  }
  __syncthreads();
  SortMap map;
  const float hi = __uint_as_float(s_hi);
  map.lo = s_lo <= s_hi ? __uint_as_float(s_lo) : 0.0f;
  map.scale = hi > map.lo ? (float)kValueBins / (hi - map.lo) : 0.0f;
  map.p_lo = s_plo <= s_phi ? (int)s_plo : 0;
  map.p_scale = s_plo < s_phi ? (float)(kSortBins - kValueBins - 1) / (float)(s_phi - s_plo) : 0.0f;
#pragma unroll 4
  for (int64_t i = t; i < n; i += kSortThreads) atomicAdd(&bins[map.bin(err_key(E[i]), P[i])], 1);
  __syncthreads();
  // exclusive prefix sums of the bins, eight of them per thread, and the fullest
  constexpr int kPer = kSortBins / kSortThreads;
  int cnt[kPer], sum = 0, most = 0;
#pragma unroll
  for (int q = 0; q < kPer; ++q) {
    cnt[q] = bins[t * kPer + q];
    sum += cnt[q];
    most = max(most, cnt[q]);
  }
  int inc = sum;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int v = __shfl_up_sync(0xffffffffu, inc, o);
    if (lane >= o) inc += v;
  }
  most = __reduce_max_sync(0xffffffffu, most);
  if (lane == 31) s_warp[t >> 5] = inc;
  if (lane == 0) atomicMax(&s_most, most);
  __syncthreads();
  int at = inc - sum;
  for (int w = 0; w < (t >> 5); ++w) at += s_warp[w];
#pragma unroll
  for (int q = 0; q < kPer; ++q) {
    bins[t * kPer + q] = at;
    at += cnt[q];
  }
  __syncthreads();
  if (s_most > kSortCap) {
    int64_t n2 = 1;
    while (n2 < n) n2 <<= 1;
    bitonic(E, P, n, n2);
    return;
  }
  // entries by bin; afterwards bins[b] is the end of bin b
  const bool whole = n <= kSortCap;
  uint64_t* by_key = whole ? sK : tmp_key + base;
  int32_t* by_p = whole ? sP : tmp_p + base;
#pragma unroll 4
  for (int64_t i = t; i < n; i += kSortThreads) {
    const uint64_t key = err_key(E[i]);
    const int32_t p = P[i];
    const int slot = atomicAdd(&bins[map.bin(key, p)], 1);
    by_key[slot] = key;
    by_p[slot] = p;
  }
  __syncthreads();
  for (int b0 = 0; b0 < kSortBins;) {
    // the window: bins b0 to b1 - 1, positions first to first + m - 1 of the list
    const int first = b0 ? bins[b0 - 1] : 0;
    int b1 = kSortBins;
    if ((int)n - first > kSortCap) {
      int above = kSortBins;  // the last b1 with bins[b1 - 1] - first <= kSortCap: at least one bin
      b1 = b0 + 1;
      while (above - b1 > 1) {
        const int mid = (b1 + above) >> 1;
        if (bins[mid - 1] - first <= kSortCap) b1 = mid; else above = mid;
      }
    }
    const int m = bins[b1 - 1] - first;
    bool crowded = false;
    for (int b = b0 + t; b < b1; b += kSortThreads)
      crowded = crowded || bins[b] - (b ? bins[b - 1] : 0) > kBinMax;
    if (!whole) {
#pragma unroll 4
      for (int i = t; i < m; i += kSortThreads) {
        sK[i] = by_key[first + i];
        sP[i] = by_p[first + i];
      }
    }
    if (__syncthreads_or(crowded)) {
      int n2 = 1;
      while (n2 < m) n2 <<= 1;
      bitonic(sK, sP, m, n2);
      for (int i = t; i < m; i += kSortThreads) {
        E[first + i] = __longlong_as_double((long long)sK[i]);
        P[first + i] = sP[i];
      }
    } else {
      for (int i = t; i < m; i += kSortThreads) {
        const uint64_t key = sK[i];
        const int32_t p = sP[i];
        const int b = map.bin(key, p);
        const int s = b ? bins[b - 1] - first : 0, e = bins[b] - first;
        int r = first + s;
        for (int j = s; j < e; ++j) r += sort_key_less(sK[j], sP[j], key, p) ? 1 : 0;
        E[r] = __longlong_as_double((long long)key);
        P[r] = p;
      }
    }
    b0 = b1;
    __syncthreads();  // before the next window's entries take their place
  }
}

cudaError_t launch_dist_group(const Cand* cand, int64_t n, int64_t G, int64_t* gcount, int64_t* goff,
                              unsigned long long* gcursor, int32_t* sp, int32_t* sg, cudaStream_t s) {
  cudaError_t err = cudaMemsetAsync(gcount, 0, sizeof(int64_t) * (size_t)G, s);
  if (err) return err;
  err = cudaMemsetAsync(gcursor, 0, sizeof(unsigned long long) * (size_t)G, s);
  if (err) return err;
  // shared-memory versions while G counters (and G reservations) fit in 48 KB
  const bool smem = G <= 4096;
  const int64_t chunk = 16384;  // candidates per block: ~2 G global atomics per 16,384 candidates at most
  const int64_t nb = (n + chunk - 1) / chunk;
  if (n > 0) {
    if (smem) {
      gene_count_smem_kernel<<<(unsigned)nb, 256, sizeof(unsigned int) * (size_t)G, s>>>(cand, n, (int)G, chunk,
                                                                                            gcount);
    } else {
      int blocks = (int)((n + 255) / 256 < 65536 ? (n + 255) / 256 : 65536);
      gene_count_kernel<<<blocks, 256, 0, s>>>(cand, n, gcount);
    }
  }
  scan_kernel<<<1, 1024, 0, s>>>(gcount, G, goff);
  if (n > 0) {
    if (smem) {
      scatter_smem_kernel<<<(unsigned)nb, 256, 12 * (size_t)G, s>>>(cand, n, (int)G, chunk, goff, gcursor, sp, sg);
    } else {
      int blocks = (int)((n + 255) / 256 < 65536 ? (n + 255) / 256 : 65536);
      scatter_kernel<<<blocks, 256, 0, s>>>(cand, n, goff, gcursor, sp, sg);
    }
  }
  return cudaGetLastError();
}

// tmp: the grouped candidates' own buffers, which nothing reads after the
// grouping (Cand is two 32-bit words, room for a key per entry)
static cudaError_t launch_segsort(const int64_t* goff, int64_t G, int32_t* sp, double* se64, const int* dirty,
                                  Cand* tmp, float* tmp_e, cudaStream_t s) {
  static_assert(sizeof(Cand) == sizeof(uint64_t) && sizeof(float) == sizeof(int32_t), "scratch of the sort");
  static std::atomic<uint64_t> attr{0};  // devices where the limit is set, shared by all contexts
  cudaError_t err = set_smem_once(attr, segsort_kernel, kSortSmem);
  if (err) return err;
  segsort_kernel<<<(unsigned)G, kSortThreads, kSortSmem, s>>>(goff, sp, se64, dirty, reinterpret_cast<uint64_t*>(tmp),
                                                              reinterpret_cast<int32_t*>(tmp_e));
  return cudaGetLastError();
}

static int grouped_blocks(int64_t n, int warps) {
  const int64_t chunks = (n + 31) / 32;
  const int64_t want = (chunks + warps - 1) / warps;
  return (int)(want < 131072 ? want : 131072);
}

static void launch_recheck_grouped(const DistInputs& in, const int32_t* sp, const int32_t* sg, int64_t n, double* se64,
                                   cudaStream_t s) {
  const int64_t chunks = (n + 31) / 32;
  if (chunks <= 4 * (int64_t)in.sms)  // at most a warp per scheduler
    recheck_grouped_kernel<1><<<(unsigned)chunks, 32, 0, s>>>(in, sp, sg, n, se64);
  else
    recheck_grouped_kernel<kRecheckWarps><<<grouped_blocks(n, kRecheckWarps), kRecheckWarps * 32, 0, s>>>(in, sp, sg, n, se64);
}

cudaError_t launch_dist_group_recheck_sort(const DistInputs& in, Cand* cand, float* cand_e, int64_t n, int64_t* gcount,
                                           int64_t* goff, unsigned long long* gcursor, int32_t* sp, int32_t* sg,
                                           double* se64, cudaStream_t s) {
  cudaError_t err = launch_dist_group(cand, n, in.G, gcount, goff, gcursor, sp, sg, s);
  if (err || n <= 0) return err;
  launch_recheck_grouped(in, sp, sg, n, se64, s);
  err = cudaGetLastError();
  if (err) return err;
  return launch_segsort(goff, in.G, sp, se64, nullptr, cand, cand_e, s);
}

cudaError_t launch_dist_group_certify_sort(const DistInputs& in, Cand* cand, float* cand_e, int64_t n, int mode, double eps,
                                           const double* eps_g, int64_t* gcount, int64_t* goff,
                                           unsigned long long* gcursor, int32_t* sp, int32_t* sg, double* se64,
                                           float4* gt, int32_t* pos, uint8_t* flag,
                                           unsigned long long* counts, int* dirty, cudaStream_t s) {
  cudaError_t err = launch_dist_group(cand, n, in.G, gcount, goff, gcursor, sp, sg, s);
  if (err) return err;
  err = cudaMemsetAsync(counts, 0, 2 * sizeof(unsigned long long), s);
  if (err) return err;
  if (n <= 0) return cudaSuccess;
  const int64_t gk = in.G * in.K;
  ff_prep_genes_kernel<<<(unsigned)((gk + 255) / 256 < 4096 ? (gk + 255) / 256 : 4096), 256, 0, s>>>(in, gt);
  const float rK = (float)(1.0 / (double)in.K);
  approx_grouped_kernel<<<grouped_blocks(n, kApproxWarps), kApproxWarps * 32, 0, s>>>(in, sp, sg, n, gt, rK, se64, pos,
                                                                                     counts);
  const int list_blocks = in.sms * 8;
  recheck_list_kernel<<<list_blocks, 128, 0, s>>>(in, sp, sg, pos, counts, se64);
  err = launch_segsort(goff, in.G, sp, se64, nullptr, cand, cand_e, s);
  if (err) return err;
  err = cudaMemsetAsync(dirty, 0, sizeof(int) * (size_t)in.G, s);
  if (err) return err;
  const int blocks = (int)((n + 255) / 256 < 65536 ? (n + 255) / 256 : 65536);
  ambiguous_kernel<<<blocks, 256, 0, s>>>(sg, goff, se64, n, mode, eps, eps_g, pos, counts + 1, flag);
  recheck_list_kernel<<<list_blocks, 128, 0, s>>>(in, sp, sg, pos, counts + 1, se64);
  run_sort_kernel<<<blocks, 256, 0, s>>>(sg, goff, flag, n, sp, se64, dirty);
  return launch_segsort(goff, in.G, sp, se64, dirty, cand, cand_e, s);
}

// ---------------------------------------------------------------------------
// accepted prefixes
// ---------------------------------------------------------------------------
__global__ void accept_len_kernel(const int64_t* goff, const double* se64, int64_t G, int mode, double eps_all,
                                  const double* eps_g, int64_t k, const float* X, const float* b0, float b1,
                                  int64_t* alen, int* n_fail, int* fail, bool approx) {
  const int64_t g = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (g >= G) return;
  const double eps = eps_g ? eps_g[g] : eps_all;
  const double* E = se64 + goff[g];
  const int64_t n = goff[g + 1] - goff[g];
  // number of finite (non-NaN) entries: NaN sorts last, and most lists have none
  // (a search of its own doubled the chain of dependent reads: 6.7 us for 4 genes)
  int64_t lo = 0, hi = n;
  if (n > 0 && E[n - 1] == E[n - 1]) lo = n;
  while (lo < hi) {
    int64_t mid = (lo + hi) >> 1;
    if (E[mid] == E[mid]) lo = mid + 1; else hi = mid;
  }
  const int64_t nn = lo;
  int64_t len;
  if (mode == 0) {
    lo = 0;
    hi = nn;
    while (lo < hi) {
      int64_t mid = (lo + hi) >> 1;
      if (E[mid] <= eps) lo = mid + 1; else hi = mid;
    }
    len = lo;
  } else {
    len = nn < k ? nn : k;
    const float x = X[g];
    bool ok;
    if (!(x < INFINITY)) {
      ok = true;  // every particle was a candidate
    } else if (len < k) {
      ok = false;
    } else {
      // every particle with err <= L had a candidate-pass error <= X
      const double L = (double)x - ((double)b0[g] + (double)b1 * (double)x);
      // certified values: the k-th error may be above its stored value by its bound
      ok = (approx ? E[k - 1] + approx_bound(E[k - 1]) : E[k - 1]) <= L;
    }
    if (!ok) {
      fail[g] = 1;
      atomicAdd(n_fail, 1);
    }
  }
  alen[g] = len;
}

cudaError_t launch_dist_accept_len(const int64_t* goff, const double* se64, int64_t G, int mode, double eps,
                                   const double* eps_g, int64_t k, const float* X, const float* b0, float b1,
                                   int64_t* alen, int* n_fail, int* fail, bool approx, cudaStream_t s) {
  if (G <= 0) return cudaSuccess;
  accept_len_kernel<<<(unsigned)((G + 127) / 128), 128, 0, s>>>(goff, se64, G, mode, eps, eps_g, k, X, b0, b1,
                                                                alen, n_fail, fail, approx);
  return cudaGetLastError();
}

__global__ void compact_kernel(const int64_t* goff, const int32_t* sp, const double* se64, const int64_t* aoff,
                               int64_t G, int64_t p_base, int64_t* idx, double* err) {
  const int64_t g = blockIdx.x;
  const int64_t src = goff[g], dst = aoff[g], n = aoff[g + 1] - aoff[g];
  for (int64_t i = threadIdx.x; i < n; i += blockDim.x) {
    idx[dst + i] = (int64_t)sp[src + i] + p_base + 1;
    if (err) err[dst + i] = se64[src + i];
  }
}

cudaError_t launch_dist_compact(const int64_t* goff, const int32_t* sp, const double* se64, const int64_t* aoff,
                                int64_t G, int64_t p_base, int64_t* idx, double* err, cudaStream_t s) {
  if (G <= 0) return cudaSuccess;
  compact_kernel<<<(unsigned)G, 256, 0, s>>>(goff, sp, se64, aoff, G, p_base, idx, err);
  return cudaGetLastError();
}

// (particle, gene) of every accepted pair, in the lists' order (grouped by gene)
__global__ void accepted_pairs_kernel(const int64_t* aoff, const int64_t* idx, int64_t G, int64_t p_base, int32_t* sp,
                                      int32_t* sg) {
  const int64_t g = blockIdx.x;
  if (g >= G) return;
  for (int64_t i = aoff[g] + threadIdx.x; i < aoff[g + 1]; i += blockDim.x) {
    sp[i] = (int32_t)(idx[i] - 1 - p_base);
    sg[i] = (int32_t)g;
  }
}

cudaError_t launch_accepted_errors(const DistInputs& in, const int64_t* aoff, const int64_t* idx, int64_t G,
                                   int64_t p_base, int64_t n, int32_t* sp, int32_t* sg, double* err, cudaStream_t s) {
  if (G <= 0 || n <= 0) return cudaSuccess;
  accepted_pairs_kernel<<<(unsigned)G, 256, 0, s>>>(aoff, idx, G, p_base, sp, sg);
  launch_recheck_grouped(in, sp, sg, n, err, s);
  return cudaGetLastError();
}

cudaError_t launch_scan(const int64_t* cnt, int64_t G, int64_t* off, cudaStream_t s) {
  scan_kernel<<<1, 1024, 0, s>>>(cnt, G, off);
  return cudaGetLastError();
}

}  // namespace abc
