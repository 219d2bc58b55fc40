// datastats.cu — the data side of the distance: the 53 statistics of every
// gene's observed per-cell counts and their bootstrap standard errors
// (scripts/data_summary_statistics.jl:1-216).  Same layout as the simulated
// statistics: [pulse mean (A), pulse FF (A), chase mean (A), chase FF (A),
// ratio (J), mean_corr (J), corr_mean (J)].
//
// Two phases: one CTA per (gene, group of resamples) forms the integer sums,
// then one thread per (gene, resample, statistic group) computes the statistics from
// them.  Resample 0 is the estimate itself, 1..n_boot are bootstrap resamples
// of the cells with replacement, drawn separately for
// the pulse cells, the chase cells and all cells (ratios and correlations), as
// the reference's get_ccp_se / get_ratio_se / get_correlation_se do.  Draw i
// of (gene, resample, family) comes from its own Philox counter, so threads
// draw independently; every statistic is computed from exact integer sums
// (n, sum x, sum x^2, sum u l per group), so the result does not depend on
// the reduction order and is bit-identical to the C oracle.  FP64 formulas
// built with -fmad=false.
#include <cuda_runtime.h>

#include <algorithm>

#include "common.cuh"
#include "distance.cuh"
#include "kernels.h"
#include "model.cuh"

namespace abc {
namespace {

constexpr int kThreads = 256;

// floor(x n / 2^64) for n < 2^32, from two 32-bit products
__device__ __forceinline__ uint32_t scaled(uint64_t x, uint32_t n) {
  const uint64_t hi = (x >> 32) * n, lo = (x & 0xffffffffu) * (uint64_t)n;
  return (uint32_t)((hi + (lo >> 32)) >> 32);
}

// positions in [0, n) of draws 2 j and 2 j + 1 of stream (seed, family, resample,
// gene): floor(x n / 2^52) of 52-bit uniform integers x, in exact integer
// arithmetic; both come from one Philox block
__device__ __forceinline__ void draw_pair(uint64_t seed, int fam, int b, int64_t g, int64_t j, int64_t n, uint32_t& p0,
                                          uint32_t& p1) {
  U4 c;
  c.x = (uint32_t)j;
  c.y = ((uint32_t)((uint64_t)j >> 32) & 0x3fffffffu) | (ST_AUX << 30);
  c.z = (uint32_t)b | ((uint32_t)(fam + 1) << 24);
  c.w = (uint32_t)g;
  const U4 o = philox4x32_10(c, (uint32_t)seed, (uint32_t)(seed >> 32));
  const uint64_t x0 = ((uint64_t)o.x << 20) | (uint64_t)(o.y >> 12), x1 = ((uint64_t)o.z << 20) | (uint64_t)(o.w >> 12);
  p0 = scaled(x0 << 12, (uint32_t)n);
  p1 = scaled(x1 << 12, (uint32_t)n);
}

// exact sample variance / covariance from integer sums, (n sxy - sx sy) /
// (n (n - 1)), with the denominator d2 and r2 = RN(1 / d2) given: the quotient
// through div_rn (correctly rounded, equal to the IEEE division)
__device__ __forceinline__ double sample_cov_r(unsigned long long n, unsigned long long sx, unsigned long long sy,
                                               unsigned long long sxy, double d2, double r2) {
  const __int128 num = (__int128)n * (__int128)sxy - (__int128)sx * (__int128)sy;
  const double x = i128_to_double(num);
  return x == 0.0 && d2 > 0.0 ? x : div_rn(x, d2, r2);  // d2 = 0 (one cell): 0 / 0 is NaN
}

// Phase 1, one CTA per (gene, resample group): the integer sums of the
// resamples b = blockIdx.y, blockIdx.y + gridDim.y, ...  The gene's cells are
// first copied into shared memory in the group-sorted order.  A resample
// only counts how often each cell is drawn (one 16-bit counter per cell, two to a
// word, one shared-memory atomic per draw); then a few lanes per (condition,
// age) group add count x (1, u, l, u^2, l^2, u l) over its cells, which are
// contiguous, in registers, and join with shuffles.  Six sums per draw through
// shared-memory atomics took 3.15 ms for 2,000 genes x 2,000 cells x 100
// resamples, this takes 2.1: the draws' Philox blocks (two draws each) are
// what is left.  Integer sums: the order does not matter.  The pulse and the
// chase draws share the counters of one pass unless both use the same cells.
constexpr size_t data_stats_smem_limit() { return 227 * 1024; }
constexpr int kMaxCount = 1 << 20;  // abc_data_stats' limit of a count

// lanes per group: the largest power of two with groups x lanes <= kThreads, at most 32
__device__ __forceinline__ int group_lanes(int groups) {
  int L = 32;
  while (L > 1 && L * groups > kThreads) L >>= 1;
  return L;
}

// threads 0 .. groups * L - 1: the sums of cells [i0, i1), joined over L lanes.
// U: 32-bit where no sum of the gene can reach 2^32 (counts up to 732 with
// 2,000 cells), 64-bit otherwise.
template <bool PAIR, typename U>
__device__ __forceinline__ void group_sums(const int2* T, const unsigned short* mult, int i0, int i1, int sub, int L,
                                           bool one, bool store, unsigned long long* out) {
  U v[6] = {0, 0, 0, 0, 0, 0};
  for (int i = i0 + sub; i < i1; i += L) {
    const U m = one ? 1u : mult[i];
    const int2 t = T[i];
    const U u = (unsigned)t.x, l = (unsigned)t.y;
    v[0] += m;
    if (PAIR) {
      const U mu = m * u, ml = m * l;
      v[1] += mu;
      v[2] += ml;
      v[3] += mu * u;
      v[4] += ml * l;
      v[5] += mu * l;
    } else {
      const U x = u + l, mx = m * x;
      v[1] += mx;
      v[2] += mx * x;
    }
  }
  for (int o = L >> 1; o > 0; o >>= 1)
#pragma unroll
    for (int q = 0; q < (PAIR ? 6 : 3); ++q) v[q] += __shfl_xor_sync(0xffffffffu, v[q], o);
  if (store)
    for (int q = 0; q < (PAIR ? 6 : 3); ++q) out[q] = v[q];
}

template <bool PAIR>
__device__ __forceinline__ void group_sums_any(bool narrow, const int2* T, const unsigned short* mult, int i0, int i1,
                                               int sub, int L, bool one, bool store, unsigned long long* out) {
  if (narrow)
    group_sums<PAIR, unsigned>(T, mult, i0, i1, sub, L, one, store, out);
  else
    group_sums<PAIR, unsigned long long>(T, mult, i0, i1, sub, L, one, store, out);
}

__device__ __forceinline__ void count_draws(const DataStatsArgs& a, unsigned* words, int fam, int b, int64_t g,
                                            int64_t base, int64_t n) {
  for (int64_t j = threadIdx.x; 2 * j < n; j += blockDim.x) {
    uint32_t p0, p1;
    draw_pair(a.seed, fam, b, g, j, n, p0, p1);
    p0 += (uint32_t)base;
    p1 += (uint32_t)base;
    // counters reach at most the number of draws, below 2^16 (data_stats_max_cells)
    atomicAdd(&words[p0 >> 1], 1u << ((p0 & 1) * 16));
    if (2 * j + 1 < n) atomicAdd(&words[p1 >> 1], 1u << ((p1 & 1) * 16));
  }
}

__global__ void __launch_bounds__(kThreads) data_sums_kernel(DataStatsArgs a, int64_t g0, unsigned long long* S_out) {
  extern __shared__ int2 T[];                                       // (u, l) per sorted cell
  const int A = a.cfg.n_ages, J = a.cfg.n_conds;
  const int nsum = 6 * A + 6 * J * A;
  const int64_t C = a.C;
  unsigned* words = reinterpret_cast<unsigned*>(T + C);             // times each cell was drawn, 16 bits each
  const unsigned short* mult = reinterpret_cast<const unsigned short*>(words);
  const int n_words = (int)((C + 1) / 2);
  const int64_t g = g0 + blockIdx.x;
  const int32_t* u = a.u + g * C;
  const int32_t* l = a.l + g * C;
  bool bad = false;
  unsigned most = 0;
  for (int64_t i = threadIdx.x; i < C; i += blockDim.x) {
    const int64_t id = a.cell_id[i];
    T[i] = make_int2(u[id], l[id]);
    const unsigned x = max((unsigned)T[i].x, (unsigned)T[i].y);
    bad = bad || x > (unsigned)kMaxCount;
    most = max(most, min(x, 1u << 20));
  }
  if (bad) *a.invalid = 1;
  // the largest sum: C draws of a cell with (u + l)^2 <= 4 most^2
  const bool narrow = __syncthreads_and(4ull * (unsigned long long)C * most * most < (1ull << 32)) != 0;
  const int cp = a.cfg.pulse_stat, cc = a.cfg.chase_stat;
  const int L2 = group_lanes(J * A), L1 = group_lanes(2 * A);
  for (int b = blockIdx.y; b <= a.n_boot; b += gridDim.y) {
    unsigned long long* out = S_out + ((int64_t)blockIdx.x * (a.n_boot + 1) + b) * nsum;
    // pulse and chase cells: per age (n, sx, sxx) at 3 A f + 3 ag
    for (int f0 = 0; f0 < 2; f0 += (cp == cc ? 1 : 2)) {
      const int f1 = cp == cc ? f0 + 1 : 2;
      __syncthreads();
      for (int i = threadIdx.x; i < n_words; i += blockDim.x) words[i] = 0u;
      __syncthreads();
      if (b > 0)
        for (int f = f0; f < f1; ++f) {
          const int cond = f == 0 ? cp : cc;
          const int64_t base = a.gstart[cond * A];
          count_draws(a, words, f, b, g, base, a.gstart[(cond + 1) * A] - base);
        }
      __syncthreads();
      const int grp = threadIdx.x / L1, f = grp / A, ag = grp - f * A;
      const bool mine = grp < 2 * A && f >= f0 && f < f1;
      const int gi = mine ? (f == 0 ? cp : cc) * A + ag : 0;
      group_sums_any<false>(narrow, T, mult, mine ? a.gstart[gi] : 0, mine ? a.gstart[gi + 1] : 0, threadIdx.x % L1, L1,
                            b == 0, mine && threadIdx.x % L1 == 0, out + 3 * grp);
    }
    // all cells: per (condition, age) (n, su, sl, suu, sll, sul)
    __syncthreads();
    for (int i = threadIdx.x; i < n_words; i += blockDim.x) words[i] = 0u;
    __syncthreads();
    if (b > 0) count_draws(a, words, 2, b, g, 0, C);
    __syncthreads();
    const int grp = threadIdx.x / L2;
    const bool mine = grp < J * A;
    group_sums_any<true>(narrow, T, mult, mine ? a.gstart[grp] : 0, mine ? a.gstart[grp + 1] : 0, threadIdx.x % L2, L2,
                         b == 0, mine && threadIdx.x % L2 == 0, out + 6 * A + 6 * grp);
  }
}

// RN(1 / n) and RN(1 / (n (n - 1))) of the sample sizes 1..C, for phase 2: a
// reciprocal each, instead of two divisions per group of every resample on the FP64 pipe
__global__ void data_recip_kernel(int64_t C, double2* recip) {
  const int64_t n = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (n < 1 || n > C) return;
  const double nd = (double)n;
  recip[n] = make_double2(1.0 / nd, 1.0 / (nd * (double)(n - 1)));
}

// a / b for b > 0 given y = RN(1 / b): div_rn, and 0 without its slow path
__device__ __forceinline__ double div_pos(double a, double b, double y) { return a == 0.0 ? a : div_rn(a, b, y); }

// Phase 2, one thread per (gene, resample, item), bound by the FP64 pipe.  First
// come the items of the conditions (ratio, mean_corr and corr_mean of condition
// it), then those of the (family, age) cells (mean and Fano factor): with both
// kinds in a warp each lane waited for the other's branch (3.2 ms against
// 1.7 for 2,000 genes x 101 resamples).
__global__ void data_stats_kernel(DataStatsArgs a, int64_t g0, int64_t ng, const unsigned long long* S_in,
                                  const double2* __restrict__ recip) {
  const int A = a.cfg.n_ages, J = a.cfg.n_conds, K = 4 * A + 3 * J;
  const int nsum = 6 * A + 6 * J * A;
  const int64_t sets = ng * (a.n_boot + 1);
  const int64_t total = sets * (2 * A + J);
  for (int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; t < total; t += (int64_t)gridDim.x * blockDim.x) {
    const bool cell = t >= sets * J;
    const int64_t q = cell ? t - sets * J : t;
    const int per = cell ? 2 * A : J;
    const int64_t gb = q / per;  // (gene - g0) * (n_boot + 1) + resample
    const int it = (int)(q - gb * per);
    const int b = (int)(gb % (a.n_boot + 1));
    const unsigned long long* Sp = S_in + gb * nsum;
    const unsigned long long* Sc = Sp + 3 * A;
    const unsigned long long* Sg = Sc + 3 * A;
    double* st = a.out + (g0 * (int64_t)(a.n_boot + 1) + gb) * K;
    if (cell) {
      // mean and Fano factor of u + l per age cluster (get_mean_ccp_data, get_ff_ccp_data)
      const int f = it / A, ag = it - (it / A) * A;
      const unsigned long long* S = f == 0 ? Sp : Sc;
      const int off = f == 0 ? 0 : 2 * A;
      const unsigned long long n = S[3 * ag];
      double m = 0.0, ff = 0.0;
      if (n > 0) {
        const double2 r = recip[n];
        const double nd = (double)n;
        m = div_pos((double)S[3 * ag + 1], nd, r.x);
        const double v = sample_cov_r(n, S[3 * ag + 1], S[3 * ag + 1], S[3 * ag + 2], nd * (double)(n - 1), r.y);
        const double eps = (m == 0.0) ? 0.0001 : 0.0;
        ff = v / (m + eps);
      }
      st[off + ag] = m;
      st[off + A + ag] = ff;
      continue;
    }
    const int j = it;
    double m1[kMaxAges], m2[kMaxAges], v1[kMaxAges], v2[kMaxAges], c12[kMaxAges], w[kMaxAges];
    unsigned long long nj = 0, suj = 0, slj = 0;
    for (int ag = 0; ag < A; ++ag) {
      const unsigned long long* S = Sg + 6 * (j * A + ag);
      nj += S[0];
      suj += S[1];
      slj += S[2];
      if (S[0] == 0) {
        m1[ag] = m2[ag] = v1[ag] = v2[ag] = c12[ag] = 0.0;
      } else {
        const double2 r = recip[S[0]];
        const double nd = (double)S[0], rn = r.x;
        m1[ag] = div_pos((double)S[1], nd, rn);
        m2[ag] = div_pos((double)S[2], nd, rn);
        const double d2 = nd * (double)(S[0] - 1), r2 = r.y;
        v1[ag] = sample_cov_r(S[0], S[1], S[1], S[3], d2, r2);
        v2[ag] = sample_cov_r(S[0], S[2], S[2], S[4], d2, r2);
        c12[ag] = sample_cov_r(S[0], S[1], S[2], S[5], d2, r2);
      }
    }
    // ratio of means (get_cond_specific_ratios)
    // nj = 0 (no cell of the condition drawn) keeps its 0 / 0
    const double njd = (double)nj, rj = nj > 0 ? recip[nj].x : INFINITY;
    const double mu = nj > 0 ? div_pos((double)suj, njd, rj) : (double)suj / njd;
    const double ml = nj > 0 ? div_pos((double)slj, njd, rj) : (double)slj / njd;
    st[4 * A + j] = (mu + ml > 0.0) ? ml / (mu + ml) : 0.0;
    // age weights: the given distribution for the estimate; for a bootstrap
    // resample the resampled cells' age fractions within the condition
    // (get_correlation_se normalises per condition)
    for (int ag = 0; ag < A; ++ag) {
      if (b == 0) {
        w[ag] = a.age_dist[ag * J + j];
      } else {
        w[ag] = nj > 0 ? div_pos((double)Sg[6 * (j * A + ag)], njd, rj) : 0.0;
      }
    }
    // get_cond_specific_correlations
    const double tv1 = wsum(w, v1, A) + wcov(m1, m1, w, A);
    const double tv2 = wsum(w, v2, A) + wcov(m2, m2, w, A);
    bool any_cov = false;
    for (int ag = 0; ag < A; ++ag) any_cov = any_cov || (c12[ag] != 0.0);
    const bool tv_ok = tv1 != 0.0 && tv2 != 0.0;
    st[4 * A + J + j] = (any_cov && tv_ok) ? wsum(w, c12, A) / sqrt(fabs(tv1 * tv2)) : 0.0;
    st[4 * A + 2 * J + j] = tv_ok ? wcov(m1, m2, w, A) / sqrt(fabs(tv1 * tv2)) : 0.0;
  }
}

// standard error over the resamples 1..n_boot of each (gene, statistic):
// sqrt(sum (v - mean)^2 / (n_boot - 1)), sums in resample order
__global__ void data_se_kernel(const double* boot, int64_t G, int K, int n_boot, double* se) {
  const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= G * K) return;
  const int64_t g = t / K;
  const int k = (int)(t - g * K);
  const double* v = boot + g * (int64_t)(n_boot + 1) * K + k;
  double s = 0.0;
  for (int b = 1; b <= n_boot; ++b) s = s + v[(int64_t)b * K];
  const double m = s / (double)n_boot;
  double q = 0.0;
  for (int b = 1; b <= n_boot; ++b) {
    const double d = v[(int64_t)b * K] - m;
    q = q + d * d;
  }
  se[t] = sqrt((1.0 / (double)(n_boot - 1)) * q);
}

}  // namespace

// (the limit of the earlier layout, which kept per-warp sums beside the 10 bytes
// per cell: calls are accepted and refused as before)
int64_t data_stats_max_cells(int n_ages, int n_conds) {
  const int64_t nsum = 6 * n_ages + 6 * n_conds * n_ages;
  return ((int64_t)data_stats_smem_limit() - (int64_t)sizeof(unsigned long long) * nsum * (kThreads / 32)) /
         (int64_t)(sizeof(int2) + sizeof(unsigned short));
}

// the sums of at most ~64 MB of (gene, resample) pairs at a time: they stay in
// L2 between the phases
static int64_t genes_at_a_time(const DevCfg& cfg, int64_t G, int n_boot, int64_t* per_gene) {
  const int64_t nsum = 6 * cfg.n_ages + 6 * cfg.n_conds * cfg.n_ages;
  *per_gene = (int64_t)(n_boot + 1) * nsum * (int64_t)sizeof(unsigned long long);
  return std::max<int64_t>(1, std::min<int64_t>(G, ((int64_t)64 << 20) / *per_gene));
}

size_t data_stats_scratch(const DevCfg& cfg, int64_t G, int n_boot, int64_t C) {
  int64_t per_gene = 0;
  const int64_t chunk = genes_at_a_time(cfg, G, n_boot, &per_gene);
  return (size_t)(chunk * per_gene) + sizeof(double2) * (size_t)(C + 1);
}

cudaError_t launch_data_stats(const DataStatsArgs& a, double* se, cudaStream_t s) {
  if (a.G <= 0) return cudaSuccess;
  const int A = a.cfg.n_ages, J = a.cfg.n_conds, K = 4 * A + 3 * J;
  const size_t smem = (size_t)a.C * sizeof(int2) + sizeof(unsigned) * (size_t)((a.C + 1) / 2);
  if (smem > data_stats_smem_limit()) return cudaErrorInvalidValue;
  if (smem > 48 * 1024) {
    cudaError_t e = cudaFuncSetAttribute(data_sums_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
  }
  int64_t per_gene = 0;
  const int64_t chunk = genes_at_a_time(a.cfg, a.G, a.n_boot, &per_gene);
  unsigned long long* S = a.sums;
  double2* recip = reinterpret_cast<double2*>(reinterpret_cast<char*>(S) + chunk * per_gene);
  cudaError_t e = cudaMemsetAsync(a.invalid, 0, sizeof(int), s);
  if (e != cudaSuccess) return e;
  data_recip_kernel<<<(unsigned)(a.C / 256 + 1), 256, 0, s>>>(a.C, recip);
  for (int64_t g0 = 0; g0 < a.G; g0 += chunk) {
    const int64_t ng = std::min<int64_t>(chunk, a.G - g0);
    // enough CTAs to fill the GPU several times over, resamples split among them
    const int64_t want = (int64_t)4 * 152 * 5;
    const int groups = (int)std::max<int64_t>(1, std::min<int64_t>(a.n_boot + 1, (want + ng - 1) / ng));
    data_sums_kernel<<<dim3((unsigned)ng, (unsigned)groups), kThreads, smem, s>>>(a, g0, S);
    const int64_t items = ng * (a.n_boot + 1) * (2 * A + J);
    const int64_t blocks = std::min<int64_t>((items + 127) / 128, 65536);
    data_stats_kernel<<<(unsigned)blocks, 128, 0, s>>>(a, g0, ng, S, recip);
    e = cudaGetLastError();
    if (e != cudaSuccess) return e;
  }
  if (a.n_boot < 2 || !se) return cudaSuccess;
  const int64_t n = a.G * K;
  data_se_kernel<<<(unsigned)((n + 255) / 256), 256, 0, s>>>(a.out, a.G, K, a.n_boot, se);
  return cudaGetLastError();
}

}  // namespace abc
