// moment.cuh — what the two modes of the moment simulation (moment.cu, FP64;
// moment_fp32.cu) share: the plan of a particle's trajectories and the kernel that
// turns their end moments into statistics.
#pragma once
#include <algorithm>
#include <cmath>

#include "common.cuh"
#include "kernels.h"
#include "model.cuh"

namespace abc {
namespace {

constexpr int NA = 10;  // 9 moments and the constant 1
constexpr int kMaxPairs = kMaxConds * kMaxAges;

// (condition, age) pairs by the start of their labelling: labelled from substep
// lo to hi, observed at end.  Substep s is the one with the midpoint t0 + (s +
// 1/2) h: the grid is aligned with every breakpoint, so midpoints are never on one.
struct MomPlan {
  int n;
  int pair[kMaxPairs], lo[kMaxPairs], hi[kMaxPairs], end[kMaxPairs];
};

inline MomPlan moment_plan(const MomArgs& a) {
  const DevCfg& cfg = a.cfg;
  const int A = cfg.n_ages;
  MomPlan plan;
  plan.n = cfg.n_conds * A;
  int lo[kMaxPairs];
  for (int t = 0; t < plan.n; ++t) {
    const double age = cfg.ages[t % A], texp = (age - cfg.pulse[t / A]) - cfg.chase[t / A];
    lo[t] = (int)std::min(std::lround((texp - cfg.t0) / a.h), std::lround((age - cfg.t0) / a.h));
    plan.pair[t] = t;
  }
  std::sort(plan.pair, plan.pair + plan.n, [&](int x, int y) { return lo[x] != lo[y] ? lo[x] < lo[y] : x < y; });
  for (int q = 0; q < plan.n; ++q) {
    const int t = plan.pair[q];
    const double age = cfg.ages[t % A], texp = (age - cfg.pulse[t / A]) - cfg.chase[t / A];
    plan.lo[q] = lo[t];
    plan.hi[q] = (int)std::lround((texp + cfg.pulse[t / A] - cfg.t0) / a.h);
    plan.end[q] = (int)std::lround((age - cfg.t0) / a.h);
  }
  return plan;
}

constexpr int kStatParticles = 8;
inline size_t stat_smem(int pairs) { return (size_t)kStatParticles * pairs * 5 * sizeof(double); }

// capture transform (model.jl:221-239) per (condition, age), then the
// statistics per condition.  moments: [n][pairs][5]; bad: per particle, nonzero
// where theta is not valid.
template <typename T>
__global__ void __launch_bounds__(128) moment_stats_kernel(MomArgs a, int64_t p0, int64_t n, const T* moments,
                                                           const T* bad_particle) {
  extern __shared__ double ds[];  // [particle][JA][5]
  const DevCfg& cfg = a.cfg;
  const int J = cfg.n_conds, A = cfg.n_ages, JA = J * A, K = 4 * A + 3 * J;
  const int64_t i0 = (int64_t)blockIdx.x * kStatParticles;
  const int np = (int)min((int64_t)kStatParticles, n - i0);
  const T* bad = bad_particle + i0;
  for (int q = threadIdx.x; q < np * JA; q += blockDim.x) {
    const int i = q / JA, t = q - i * JA;
    if (bad[i] != T(0)) continue;
    const int j = t / A, ai = t - (t / A) * A;
    const double* bm = a.beta_mom + ((j < a.n_pulse_conds ? 0 : 1) * A + ai) * 3;
    const double mb = bm[0], m2 = bm[1], vb = bm[2];
    double sm[5];
#pragma unroll
    for (int e = 0; e < 5; ++e) sm[e] = moments[(i0 * JA + q) * 5 + e];
    double* d = ds + (size_t)q * 5;
    d[0] = sm[0] * mb;
    d[1] = sm[1] * mb;
    d[2] = ((mb - m2) * sm[0] + vb * (sm[0] * sm[0] + sm[2])) + mb * mb * sm[2];
    d[4] = ((mb - m2) * sm[1] + vb * (sm[1] * sm[1] + sm[4])) + mb * mb * sm[4];
    d[3] = vb * (sm[0] * sm[1] + sm[3]) + mb * mb * sm[3];
    if (a.moments)
#pragma unroll
      for (int e = 0; e < 5; ++e) a.moments[((p0 + i0) * JA + q) * 5 + e] = sm[e];
  }
  __syncthreads();
  for (int q = threadIdx.x; q < np * J; q += blockDim.x) {
    const int i = q / J, j = q - i * J;
    if (bad[i] == T(0))
      stats_from_moments_cond(cfg, ds + (size_t)i * JA * 5, a.age_dist, a.stats + (p0 + i0 + i) * K, j);
  }
  for (int q = threadIdx.x; q < np * K; q += blockDim.x) {
    const int i = q / K;
    if (bad[i] == T(0)) continue;
    a.stats[(p0 + i0) * K + q] = NAN;
    if (q == i * K) atomicOr(a.status, 1);
  }
}

// particles per chunk: propagators of at most ~256 MB
inline int64_t moment_chunk(int64_t P, int nsub, size_t prop_bytes) {
  const int64_t bytes = (int64_t)2 * nsub * (int64_t)prop_bytes;
  return std::max<int64_t>(1, std::min<int64_t>(P, ((int64_t)256 << 20) / bytes));
}

}  // namespace
}  // namespace abc
