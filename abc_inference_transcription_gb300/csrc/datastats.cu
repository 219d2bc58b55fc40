// datastats.cu — the data side of the distance: the 53 statistics of every
// gene's observed per-cell counts and their bootstrap standard errors
// (scripts/data_summary_statistics.jl:1-216).  Same layout as the simulated
// statistics: [pulse mean (A), pulse FF (A), chase mean (A), chase FF (A),
// ratio (J), mean_corr (J), corr_mean (J)].
//
// Two phases: one CTA per (gene, group of resamples) forms the integer sums,
// then one thread per (gene, resample, statistic group) computes the statistics from
// them, a chunk of genes behind.  Resample 0 is the estimate itself, 1..n_boot are bootstrap resamples
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
#include <atomic>

#include "common.cuh"
#include "distance.cuh"
#include "kernels.h"
#include "model.cuh"
#include "smem_attr.h"

namespace abc {
namespace {

constexpr int kThreads = 256;

struct DrawKeys {
  uint32_t k[20];
};

// positions in [0, n) of draws 2 j and 2 j + 1 of stream (seed, family, resample,
// gene): floor(x n / 2^52) of 52-bit uniform integers x (the top bits of a word
// pair), in exact integer arithmetic; both come from one Philox block
__device__ __forceinline__ uint32_t scaled(uint32_t hi, uint32_t lo, uint32_t n) {
  return (uint32_t)(((uint64_t)hi * n + __umulhi(lo & 0xfffff000u, n)) >> 32);
}
// (Philox4x32-10 with the round keys from the launch's parameters: formed from the seed
// by every thread, they were 18 of a block's 60 instructions)
__device__ __forceinline__ void draw_pair(const DrawKeys& keys, int fam, int b, int64_t g, uint32_t j, uint32_t n,
                                          uint32_t& p0, uint32_t& p1) {
  U4 c;
  c.x = j;
  c.y = ST_AUX << 30;
  c.z = (uint32_t)b | ((uint32_t)(fam + 1) << 24);
  c.w = (uint32_t)g;
#pragma unroll
  for (int r = 0; r < 10; ++r) {
    const uint64_t m0 = (uint64_t)0xD2511F53u * (uint64_t)c.x, m1 = (uint64_t)0xCD9E8D57u * (uint64_t)c.z;
    c = U4{(uint32_t)(m1 >> 32) ^ c.y ^ keys.k[2 * r], (uint32_t)m1, (uint32_t)(m0 >> 32) ^ c.w ^ keys.k[2 * r + 1],
           (uint32_t)m0};
  }
  p0 = scaled(c.x, c.y, n);
  p1 = scaled(c.z, c.w, n);
}

// Phase 1, one CTA per (gene, resample group): the integer sums of the
// resamples b = blockIdx.y, blockIdx.y + gridDim.y, ...  The gene's cells are
// first copied into shared memory in the group-sorted order.  A resample
// only counts how often each cell is drawn (a word per cell: draws from all cells in
// the low half, from the pulse or chase cells in the high half, one shared-memory
// atomic per draw); then a few lanes per (condition, age) group add count x
// (1, u, l, u^2, l^2, u l) over its cells, which are contiguous, in registers,
// and join with shuffles.  Six sums per draw through shared-memory atomics took
// 3.15 ms for 2,000 genes x 2,000 cells x 100 resamples, a pass of its own per family of
// draws 2.1, this takes 1.75: bound by instruction issue, half of it the draws'
// Philox blocks (two draws each).  Integer sums: the order does not matter.
constexpr size_t data_stats_smem_limit() { return 227 * 1024; }
constexpr int kMaxCount = 1 << 20;  // abc_data_stats' limit of a count

// log2 of the lanes per group: the largest power of two with groups x lanes <= kThreads, at most 32
__device__ __forceinline__ int log_group_lanes(int groups) {
  int lg = 5;
  while (lg > 0 && (groups << lg) > kThreads) lg--;
  return lg;
}

// a cell's (u, l) in the group-sorted order: from the copy, or through the
// order where the copy does not fit beside the counters
struct Cells {
  const int2* T;
  const uint32_t* id;
  const int32_t *u, *l;
  __device__ __forceinline__ int2 operator[](int i) const {
    if (T) return T[i];
    const uint32_t c = id[i];
    return make_int2(u[c], l[c]);
  }
};

// threads 0 .. groups * L - 1: the sums of cells [i0, i1), joined over L lanes.
// U: 32-bit where no sum of the gene can reach 2^32 (counts up to 732 with
// 2,000 cells), 64-bit otherwise.
template <bool PAIR, typename U>
__device__ __forceinline__ void group_sums(const Cells& T, const unsigned* drawn, int i0, int i1, int sub, int L,
                                           bool one, bool store, unsigned long long* out) {
  U v[6] = {0, 0, 0, 0, 0, 0};
  for (int i = i0 + sub; i < i1; i += L) {
    const U m = one ? 1u : PAIR ? drawn[i] & 0xffffu : drawn[i] >> 16;
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
__device__ __forceinline__ void group_sums_any(bool narrow, const Cells& T, const unsigned* drawn, int i0, int i1,
                                               int sub, int L, bool one, bool store, unsigned long long* out) {
  if (narrow)
    group_sums<PAIR, unsigned>(T, drawn, i0, i1, sub, L, one, store, out);
  else
    group_sums<PAIR, unsigned long long>(T, drawn, i0, i1, sub, L, one, store, out);
}

// n draws among the cells from base on, `inc` added to each one's word.  The
// first pair falls to thread `first`, so that the families of a resample share the
// threads evenly; returns the thread after the last.  Each half of a word reaches
// at most n, below 2^16 (data_stats_max_cells).
__device__ __forceinline__ int count_draws(const DrawKeys& keys, unsigned* drawn, int fam, int b, int64_t g, int base,
                                           int n, unsigned inc, int first) {
  const int pairs = (n + 1) / 2;
  for (int j = (threadIdx.x - first) & (kThreads - 1); j < pairs; j += kThreads) {
    uint32_t p0, p1;
    draw_pair(keys, fam, b, g, (uint32_t)j, (uint32_t)n, p0, p1);
    atomicAdd(&drawn[base + p0], inc);
    if (2 * j + 1 < n) atomicAdd(&drawn[base + p1], inc);
  }
  return (first + pairs) & (kThreads - 1);
}

__device__ __forceinline__ void sums_block(const DataStatsArgs& a, unsigned* drawn, bool copy, const DrawKeys& keys,
                                           int64_t g0, int gene, int b0, int b_step, unsigned long long* S_out) {
  const int A = a.cfg.n_ages, J = a.cfg.n_conds;
  const int nsum = 6 * A + 6 * J * A;
  const int C = (int)a.C;
  int2* T = copy ? reinterpret_cast<int2*>(drawn + (C + 1) / 2 * 2) : nullptr;
  const int64_t g = g0 + gene;
  const int32_t* u = a.u + g * C;
  const int32_t* l = a.l + g * C;
  bool bad = false;
  unsigned most = 0;
  for (int i = threadIdx.x; i < C; i += kThreads) {
    const uint32_t id = a.cell_id[i];
    const int2 t = make_int2(u[id], l[id]);
    if (T) T[i] = t;
    const unsigned x = max((unsigned)t.x, (unsigned)t.y);
    bad = bad || x > (unsigned)kMaxCount;
    most = max(most, min(x, 1u << 20));
  }
  if (bad) *a.invalid = 1;
  // the largest sum: C draws of a cell with (u + l)^2 <= 4 most^2
  const bool narrow = __syncthreads_and(4ull * (unsigned long long)C * most * most < (1ull << 32)) != 0;
  const Cells cells = {T, a.cell_id, u, l};
  const int cp = a.cfg.pulse_stat, cc = a.cfg.chase_stat;
  // this thread's (condition, age) group, and its (family, age) group of the pulse or chase cells
  const int lg2 = log_group_lanes(J * A), lg1 = log_group_lanes(2 * A);
  const int grp2 = threadIdx.x >> lg2, grp1 = threadIdx.x >> lg1;
  const bool in2 = grp2 < J * A, in1 = grp1 < 2 * A;
  const int s2 = in2 ? a.gstart[grp2] : 0, e2 = in2 ? a.gstart[grp2 + 1] : 0;
  const int fam1 = grp1 < A ? 0 : 1, gi = in1 ? (fam1 ? cc : cp) * A + grp1 - fam1 * A : 0;
  const int s1 = in1 ? a.gstart[gi] : 0, e1 = in1 ? a.gstart[gi + 1] : 0;
  const int base[2] = {a.gstart[cp * A], a.gstart[cc * A]};
  const int size[2] = {a.gstart[(cp + 1) * A] - base[0], a.gstart[(cc + 1) * A] - base[1]};
  for (int b = b0; b <= a.n_boot; b += b_step) {
    unsigned long long* out = S_out + ((int64_t)gene * (a.n_boot + 1) + b) * nsum;
    // the chase draws share the pass of the others unless they fall on the pulse cells
    for (int pass = 0; pass < (cp == cc ? 2 : 1); ++pass) {
      const int f0 = pass, f1 = cp == cc ? pass + 1 : 2;
      __syncthreads();
      if (b > 0) {
        for (int i = threadIdx.x; i < C; i += kThreads) drawn[i] = 0u;
        __syncthreads();
        int first = pass == 0 ? count_draws(keys, drawn, 2, b, g, 0, C, 1u, 0) : 0;
        for (int f = f0; f < f1; ++f)
          first = count_draws(keys, drawn, f, b, g, base[f], size[f], 1u << 16, first);
        __syncthreads();
      }
      // all cells: per (condition, age) (n, su, sl, suu, sll, sul)
      if (pass == 0) {
        const int sub = threadIdx.x & ((1 << lg2) - 1);
        group_sums_any<true>(narrow, cells, drawn, s2, e2, sub, 1 << lg2, b == 0, in2 && sub == 0,
                             out + 6 * A + 6 * grp2);
      }
      // pulse and chase cells: per age (n, sx, sxx) at 3 A f + 3 ag
      const bool mine = in1 && fam1 >= f0 && fam1 < f1;
      const int sub = threadIdx.x & ((1 << lg1) - 1);
      group_sums_any<false>(narrow, cells, drawn, s1, mine ? e1 : s1, sub, 1 << lg1, b == 0, mine && sub == 0,
                            out + 3 * grp1);
    }
  }
}

// n, n (n - 1) and their correctly rounded reciprocals for the sample sizes 1..C, for
// phase 2: a load each, instead of a conversion or a division on the FP64 pipe
struct SizeTerms {
  double n, rn, d2, r2;
};
__global__ void data_recip_kernel(int64_t C, SizeTerms* terms) {
  const int64_t n = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (n < 1 || n > C) return;
  const double nd = (double)n, d2 = nd * (double)(n - 1);
  terms[n] = SizeTerms{nd, 1.0 / nd, d2, 1.0 / d2};
}

// Quotients of integer sums, correctly rounded through div_rn (equal to the
// IEEE division).  Zeros are told by the integers: an FP64 comparison takes the
// pipe that bounds this phase as long as a multiplication.
__device__ __forceinline__ double mean_r(unsigned long long s, double n, double rn) {
  return s == 0 ? 0.0 : div_rn((double)s, n, rn);
}
// exact sample variance / covariance (n sxy - sx sy) / (n (n - 1)); nonzero: whether
// it is not 0 (one cell gives 0 / 0 = NaN, which is not)
__device__ __forceinline__ double cov_r(unsigned long long n, unsigned long long sx, unsigned long long sy,
                                        unsigned long long sxy, const SizeTerms& t, bool& nonzero) {
  const __int128 num = (__int128)n * (__int128)sxy - (__int128)sx * (__int128)sy;
  nonzero = num != 0 || n <= 1;
  return nonzero ? div_rn(i128_to_double(num), t.d2, t.r2) : 0.0;
}
__device__ __forceinline__ bool is_zero(double x) { return (__double_as_longlong(x) << 1) == 0; }

// Phase 2, one thread per (gene, resample, item), bound by the FP64 pipe.  First
// come the items of the conditions (ratio, mean_corr and corr_mean of condition
// it), then those of the (family, age) cells (mean and Fano factor): with both
// kinds in a warp each lane waited for the other's branch (3.2 ms for 2,000 genes
// x 101 resamples, 1.7 by kind, 1.26 without the comparisons, conversions and the
// second square root).
__device__ __forceinline__ void stats_item(const DataStatsArgs& a, int64_t g0, int64_t ng,
                                           const unsigned long long* S_in, const SizeTerms* __restrict__ terms,
                                           int64_t t) {
  const int A = a.cfg.n_ages, J = a.cfg.n_conds, K = 4 * A + 3 * J;
  const int nsum = 6 * A + 6 * J * A;
  const int64_t sets = ng * (a.n_boot + 1);
  if (t >= sets * (2 * A + J)) return;
  {
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
    bool nonzero;
    if (cell) {
      // mean and Fano factor of u + l per age cluster (get_mean_ccp_data, get_ff_ccp_data)
      const int f = it / A, ag = it - (it / A) * A;
      const unsigned long long* S = f == 0 ? Sp : Sc;
      const int off = f == 0 ? 0 : 2 * A;
      const unsigned long long n = S[3 * ag], sx = S[3 * ag + 1];
      double m = 0.0, ff = 0.0;
      if (n > 0) {
        const SizeTerms r = terms[n];
        m = mean_r(sx, r.n, r.rn);
        ff = cov_r(n, sx, sx, S[3 * ag + 2], r, nonzero) / (sx == 0 ? 0.0001 : m);
      }
      st[off + ag] = m;
      st[off + A + ag] = ff;
      return;
    }
    const int j = it;
    double m1[kMaxAges], m2[kMaxAges], v1[kMaxAges], v2[kMaxAges], c12[kMaxAges], w[kMaxAges];
    unsigned long long nj = 0, suj = 0, slj = 0;
    bool any_cov = false;
    for (int ag = 0; ag < A; ++ag) {
      const unsigned long long* S = Sg + 6 * (j * A + ag);
      nj += S[0];
      suj += S[1];
      slj += S[2];
      if (S[0] == 0) {
        m1[ag] = m2[ag] = v1[ag] = v2[ag] = c12[ag] = 0.0;
      } else {
        const SizeTerms r = terms[S[0]];
        m1[ag] = mean_r(S[1], r.n, r.rn);
        m2[ag] = mean_r(S[2], r.n, r.rn);
        v1[ag] = cov_r(S[0], S[1], S[1], S[3], r, nonzero);
        v2[ag] = cov_r(S[0], S[2], S[2], S[4], r, nonzero);
        c12[ag] = cov_r(S[0], S[1], S[2], S[5], r, nonzero);
        any_cov = any_cov || nonzero;
      }
    }
    // ratio of means (get_cond_specific_ratios); 0 without a molecule or a cell
    const double njd = nj > 0 ? terms[nj].n : 0.0, rj = nj > 0 ? terms[nj].rn : 0.0;
    double ratio = 0.0;
    if (suj + slj > 0) {
      const double ml = mean_r(slj, njd, rj);
      ratio = ml / (mean_r(suj, njd, rj) + ml);
    }
    st[4 * A + j] = ratio;
    // age weights: the given distribution for the estimate; for a bootstrap
    // resample the resampled cells' age fractions within the condition
    // (get_correlation_se normalises per condition)
    for (int ag = 0; ag < A; ++ag)
      w[ag] = b == 0 ? a.age_dist[ag * J + j] : nj > 0 ? mean_r(Sg[6 * (j * A + ag)], njd, rj) : 0.0;
    // get_cond_specific_correlations: wsum(w, v) + wcov(m, m) and wcov(m1, m2), the
    // means and deviations of the three wcov formed once
    const double mx = wsum(w, m1, A), my = wsum(w, m2, A);
    double s11 = 0.0, s22 = 0.0, s12 = 0.0;
    for (int ag = 0; ag < A; ++ag) {
      const double dx = m1[ag] - mx, dy = m2[ag] - my;
      const double p11 = w[ag] * (dx * dx), p22 = w[ag] * (dy * dy), p12 = w[ag] * (dx * dy);
      s11 = ag ? s11 + p11 : p11;
      s22 = ag ? s22 + p22 : p22;
      s12 = ag ? s12 + p12 : p12;
    }
    const double tv1 = wsum(w, v1, A) + s11;
    const double tv2 = wsum(w, v2, A) + s22;
    double mean_corr = 0.0, corr_mean = 0.0;
    if (!is_zero(tv1) && !is_zero(tv2)) {
      const double sd = sqrt(fabs(tv1 * tv2));
      if (any_cov) mean_corr = wsum(w, c12, A) / sd;
      corr_mean = s12 / sd;
    }
    st[4 * A + J + j] = mean_corr;
    st[4 * A + 2 * J + j] = corr_mean;
  }
}

// Both phases in one launch: the sums of one chunk of genes beside the statistics of
// the chunk before, blocks of the two kinds in turn.  The sums are bound by
// instruction issue, the statistics by the FP64 pipe, so they share a
// multiprocessor well (2,000 genes x 2,000 cells x 100
// resamples, the whole call: 3.42 ms in launches of their own, 2.82 here; five blocks a
// multiprocessor, four took 3.05).
struct DataChunk {
  int64_t g0, n;          // first gene, genes (0: none)
  unsigned long long* S;  // [n][n_boot + 1][nsum]
};
__global__ void __launch_bounds__(kThreads, 5) data_phases_kernel(const __grid_constant__ DataStatsArgs a,
                                                                  const __grid_constant__ DrawKeys keys, bool copy,
                                                                  DataChunk sums, int groups, DataChunk stats,
                                                                  int64_t stats_blocks, const SizeTerms* terms) {
  extern __shared__ unsigned drawn[];  // per sorted cell, then the copy of the cells
  // of the first b blocks, b stats_blocks / gridDim.x are of the second kind
  const int64_t b = blockIdx.x, before = b * stats_blocks / gridDim.x;
  if ((b + 1) * stats_blocks / gridDim.x > before) {
    stats_item(a, stats.g0, stats.n, stats.S, terms, before * kThreads + threadIdx.x);
  } else {
    const int64_t i = b - before;
    sums_block(a, drawn, copy, keys, sums.g0, (int)(i / groups), (int)(i % groups), groups, sums.S);
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

// the sums of at most ~64 MB of (gene, resample) pairs at a time, twice
static int64_t genes_at_a_time(const DevCfg& cfg, int64_t G, int n_boot, int64_t* per_gene) {
  const int64_t nsum = 6 * cfg.n_ages + 6 * cfg.n_conds * cfg.n_ages;
  *per_gene = (int64_t)(n_boot + 1) * nsum * (int64_t)sizeof(unsigned long long);
  return std::max<int64_t>(1, std::min<int64_t>(G, ((int64_t)64 << 20) / *per_gene));
}

size_t data_stats_scratch(const DevCfg& cfg, int64_t G, int n_boot, int64_t C) {
  int64_t per_gene = 0;
  const int64_t chunk = genes_at_a_time(cfg, G, n_boot, &per_gene);
  return (size_t)(2 * chunk * per_gene) + sizeof(SizeTerms) * (size_t)(C + 1);
}

cudaError_t launch_data_stats(const DataStatsArgs& a, double* se, cudaStream_t s) {
  if (a.G <= 0) return cudaSuccess;
  const int A = a.cfg.n_ages, J = a.cfg.n_conds, K = 4 * A + 3 * J;
  size_t smem = sizeof(unsigned) * (size_t)((a.C + 1) / 2 * 2);
  const bool copy = smem + (size_t)a.C * sizeof(int2) <= data_stats_smem_limit();
  if (copy) smem += (size_t)a.C * sizeof(int2);
  if (smem > data_stats_smem_limit()) return cudaErrorInvalidValue;
  static std::atomic<uint64_t> attr{0};  // the largest size sets the limit once per device, for all contexts
  cudaError_t e = set_smem_once(attr, data_phases_kernel, (int)data_stats_smem_limit());
  if (e != cudaSuccess) return e;
  int64_t per_gene = 0;
  const int64_t chunk = genes_at_a_time(a.cfg, a.G, a.n_boot, &per_gene);
  unsigned long long* S = a.sums;
  SizeTerms* terms = reinterpret_cast<SizeTerms*>(reinterpret_cast<char*>(S) + 2 * chunk * per_gene);
  e = cudaMemsetAsync(a.invalid, 0, sizeof(int), s);
  if (e != cudaSuccess) return e;
  DrawKeys keys;
  for (int r = 0; r < 10; ++r) {  // Weyl sequences of the Philox key
    keys.k[2 * r] = (uint32_t)a.seed + (uint32_t)r * 0x9E3779B9u;
    keys.k[2 * r + 1] = (uint32_t)(a.seed >> 32) + (uint32_t)r * 0xBB67AE85u;
  }
  data_recip_kernel<<<(unsigned)(a.C / 256 + 1), 256, 0, s>>>(a.C, terms);
  DataChunk before{0, 0, nullptr};
  for (int64_t g0 = 0; g0 < a.G || before.n > 0; g0 += chunk) {
    const int64_t ng = std::max<int64_t>(0, std::min<int64_t>(chunk, a.G - g0));
    const DataChunk now{g0, ng, S + (g0 / chunk % 2) * (chunk * per_gene / (int64_t)sizeof(unsigned long long))};
    // enough CTAs to fill the GPU several times over, resamples split among them
    const int64_t want = (int64_t)4 * a.sms * 5;
    const int groups = ng ? (int)std::max<int64_t>(1, std::min<int64_t>(a.n_boot + 1, (want + ng - 1) / ng)) : 1;
    const int64_t items = before.n * (a.n_boot + 1) * (2 * A + J);
    const int64_t stats_blocks = (items + kThreads - 1) / kThreads;
    data_phases_kernel<<<(unsigned)(ng * groups + stats_blocks), kThreads, smem, s>>>(a, keys, copy, now, groups, before,
                                                                                   stats_blocks, terms);
    e = cudaGetLastError();
    if (e != cudaSuccess) return e;
    before = now;
  }
  if (a.n_boot < 2 || !se) return cudaSuccess;
  const int64_t n = a.G * K;
  data_se_kernel<<<(unsigned)((n + 255) / 256), 256, 0, s>>>(a.out, a.G, K, a.n_boot, se);
  return cudaGetLastError();
}

}  // namespace abc
