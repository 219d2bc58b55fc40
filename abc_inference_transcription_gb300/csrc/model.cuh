// model.cuh — per-particle model records and the statistics aggregation.
//
// Reference (paths inside pthomaslab/abc_inference_transcription):
//   theta layout  hcat(kon, koff, alpha, gamma, lambda)  scripts/abc_simulation.jl:10
//   varying rate  get_vary_map / get_rate               scripts/model.jl:1-43
//   statistics    abc_sim                               scripts/abc_simulation.jl:23-46
//                 weighted_cov                          scripts/data_summary_statistics.jl:179-181
#pragma once
#include <cmath>
#include "common.cuh"

namespace abc {

constexpr int kMaxSteps = 8;
constexpr int kMaxAges = 8;
constexpr int kMaxConds = 16;

// Time grid and options, passed by value to every kernel.
struct DevCfg {
  double cycle, step_len, t0;
  double ages[kMaxAges];
  double pulse[kMaxConds];
  double chase[kMaxConds];
  int64_t event_cap;
  int n_steps, n_ages, n_conds, splicing, scaling_column, pulse_stat, chase_stat, npar;
  // Breakpoint grid (dcfg_set_grid): when every time above is an integer
  // multiple of quantum = 2^-e, the same times in quanta, so that the
  // production SSA places breakpoints with exact integer arithmetic.
  int grid_ok;
  float quantum;
  int32_t t0_q, cycle_q, step_q;
  int32_t ages_q[kMaxAges], pulse_q[kMaxConds], chase_q[kMaxConds];
};

// Host: find the coarsest quantum 2^-e (e = 0..20) of which t0, the cycle, the
// age step, every age, pulse and chase are exact integer multiples, with every
// breakpoint time (at most a few cycles) below 2^30 quanta; grid_ok = 0 if none.
inline void dcfg_set_grid(DevCfg& d) {
  d.grid_ok = 0;
  double horizon = std::fabs(d.t0) + 2.0 * d.cycle;
  for (int a = 0; a < d.n_ages; ++a) horizon = std::fmax(horizon, std::fabs(d.ages[a]) + std::fabs(d.t0));
  for (int e = 0; e <= 20; ++e) {
    const double sc = std::ldexp(1.0, e);
    auto ok = [&](double t) {
      const double x = t * sc;
      return x == std::floor(x) && std::fabs(x) < 1073741824.0;
    };
    bool all = ok(d.t0) && ok(d.cycle) && ok(d.step_len) && horizon * sc < 1073741824.0;
    for (int a = 0; a < d.n_ages && all; ++a) all = ok(d.ages[a]);
    for (int j = 0; j < d.n_conds && all; ++j) all = ok(d.pulse[j]) && ok(d.chase[j]);
    if (!all) continue;
    d.grid_ok = 1;
    d.quantum = (float)std::ldexp(1.0, -e);
    d.t0_q = (int32_t)(d.t0 * sc);
    d.cycle_q = (int32_t)(d.cycle * sc);
    d.step_q = (int32_t)(d.step_len * sc);
    for (int a = 0; a < kMaxAges; ++a) d.ages_q[a] = a < d.n_ages ? (int32_t)(d.ages[a] * sc) : 0;
    for (int j = 0; j < kMaxConds; ++j) {
      d.pulse_q[j] = j < d.n_conds ? (int32_t)(d.pulse[j] * sc) : 0;
      d.chase_q[j] = j < d.n_conds ? (int32_t)(d.chase[j] * sc) : 0;
    }
    return;
  }
}

// FP64 particle record (rates are 10^theta).
struct PRec {
  double kon[kMaxSteps], alp[kMaxSteps], gam[kMaxSteps], amax[kMaxSteps];
  double koff, lam, beta, scal;
  double g0, u0, s0;  // means at the start of a cycle (SSA initial state)
  double c0, v0;      // Cov(G, u) and Var u there (no splicing)
  double cost;        // expected fired events per trajectory (work estimate)
};

// FP32 copy of the rates for the production SSA, in log2 units: every rate
// (kon, alp, gam, amax, koff, beta) times log2 e; lam (a probability) and
// scal (an exponent) as they are.
struct PRecF {
  float kon[kMaxSteps], alp[kMaxSteps], gam[kMaxSteps], amax[kMaxSteps];
  float koff, lam, beta, scal;
};

// ---------------------------------------------------------------------------
// Initial state: periodic solution of the mean equations of (G, first mRNA
// species, spliced species) over one cycle with division, solved as the fixed
// point of the affine cycle map.  Exact exponential sub-steps with the
// substep-averaged source (16 per age step).
// ---------------------------------------------------------------------------
constexpr int kIcSub = 16;

ABC_HD void phi_pair(double z, double& e, double& ph) {
  e = xexp(-z);
  ph = (z > 1e-6) ? (1.0 - e) / z : 1.0 - 0.5 * z;
}

ABC_HD void mean_cycle(const DevCfg& cfg, const PRec& R, double& G, double& uu, double& us) {
  const int S = cfg.n_steps;
  const double T = cfg.cycle;
  const double h = (T / (double)S) / (double)kIcSub;
  for (int k = 0; k < S; ++k) {
    double kG = R.kon[k] + R.koff;
    double Ginf = R.kon[k] / kG;
    double eG, phG, eu, phu, es = 0.0, phs = 0.0;
    phi_pair(kG * h, eG, phG);
    double ku = cfg.splicing ? R.beta : R.gam[k];
    phi_pair(ku * h, eu, phu);
    if (cfg.splicing) phi_pair(R.gam[k] * h, es, phs);
    for (int i = 0; i < kIcSub; ++i) {
      double ph = ((double)(k * kIcSub + i) + 0.5) * h;
      double a = R.alp[k] * xpow(1.0 + ph / T, R.scal);
      double Gavg = Ginf + (G - Ginf) * phG;
      double Gn = Ginf + (G - Ginf) * eG;
      double uun = uu * eu + ((a * Gavg) * h) * phu;
      double usn = 0.0;
      if (cfg.splicing) usn = us * es + ((R.beta * (0.5 * (uu + uun))) * h) * phs;
      G = Gn;
      uu = uun;
      us = usn;
    }
  }
  uu = uu * 0.5;
  us = us * 0.5;
}

// b: the cycle map of (0, 0, 0); c[i]: of the i-th unit vector
ABC_HD void solve_initial_means(const DevCfg& cfg, const double b[3], const double c[3][3], PRec& R) {
  double mGG = c[0][0] - b[0];
  double muG = c[0][1] - b[1], muu = c[1][1] - b[1];
  double msG = c[0][2] - b[2], msu = c[1][2] - b[2], mss = c[2][2] - b[2];
  double g = b[0] / (1.0 - mGG);
  double u = (b[1] + muG * g) / (1.0 - muu);
  double s = cfg.splicing ? ((b[2] + msG * g) + msu * u) / (1.0 - mss) : 0.0;
  if (!(g > 0.0)) g = 0.0;
  if (g > 1.0) g = 1.0;
  if (!(u > 0.0)) u = 0.0;
  if (!(s > 0.0)) s = 0.0;
  R.g0 = g;
  R.u0 = u;
  R.s0 = s;
}

// ---------------------------------------------------------------------------
// Initial state without splicing: the periodic solution, at the start of a
// cycle (after division), of the unlabelled moments x = (E G, E u, Cov(G,u),
// Var u) of the reaction network (model.jl:67-86 with lambda = 0) under the
// division map (model.jl:98-111: Cov/2, Var/4 + E/4, E/2), i.e. the state
// transient_phase converges to (model.jl:114-142).
//   E G' = kon - (kon + koff) E G
//   E u' = alpha(t) E G - gamma E u
//   C'   = alpha(t) E G (1 - E G) - (kon + koff + gamma) C
//   V'   = alpha(t) E G + gamma E u + 2 alpha(t) C - 2 gamma V
// Exponential sub-steps (16 per age step) with the sources averaged over the
// sub-step.  E G is periodic by itself; with it fixed, the cycle map of
// (E u, C, V) is affine with a lower-triangular matrix, solved directly
// (initial_moments_lanes in kernels_fp64.cu).
// ---------------------------------------------------------------------------

// Unspliced count at the start of a trajectory, given the gene state G drawn
// with probability g0: conditional mean E[u | G] = u0 + c0 / g0 (G = 1) or
// u0 - c0 / (1 - g0) (G = 0), and within-state variance F E[u | G] with the
// Fano factor F = (v0 - c0^2 / (g0 (1 - g0))) / u0, so that E u, Var u and
// Cov(G, u) are those of the periodic solution.  Drawn as a zero-inflated
// Poisson (0 with probability 1 - w, else Poisson(mu / w), w = mu / (mu + F - 1))
// when F > 1, a Poisson(mu) otherwise.  wz: a 32-bit uniform word for the
// zero inflation; aux: the trajectory's auxiliary stream.
ABC_HD int64_t initial_count(const PRec& R, int G, uint32_t wz, Rng& aux) {
  const double g = R.g0, m = R.u0, c = R.c0, v = R.v0;
  double mu = m, vr = v;
  if (g > 0.0 && g < 1.0) {
    mu = G ? m + c / g : m - c / (1.0 - g);
    vr = v - (c * c) / (g * (1.0 - g));
  }
  if (!(mu > 0.0)) return 0;
  const double F = (m > 0.0 && vr > 0.0) ? vr / m : 0.0;
  double lam = mu;
  if (F > 1.0) {
    const double w = mu / (mu + (F - 1.0));
    if (!((double)wz * ABC_TWO_M32 < w)) return 0;
    lam = mu / w;
  }
  return poisson(aux, lam);
}

// theta -> rates of the record (the moment ODE's; the SSA's setup_kernel also
// fills the initial state and work estimate); returns 0 or a negative abc_status.
ABC_HD int parse_theta(const DevCfg& cfg, int model, const double* th, PRec& R) {
  const int S = cfg.n_steps;
  int i = 0;
  double lk[kMaxSteps], la[kMaxSteps], lg[kMaxSteps];
  if (model == 3) {
    for (int k = 0; k < S; ++k) lk[k] = th[i++];
  } else {
    double v = th[i++];
    for (int k = 0; k < S; ++k) lk[k] = v;
  }
  double lkoff = th[i++];
  if (model == 4) {
    for (int k = 0; k < S; ++k) la[k] = th[i++];
  } else {
    double v = th[i++];
    for (int k = 0; k < S; ++k) la[k] = v;
  }
  if (model == 5) {
    for (int k = 0; k < S; ++k) lg[k] = th[i++];
  } else {
    double v = th[i++];
    for (int k = 0; k < S; ++k) lg[k] = v;
  }
  double llam = th[i++];
  R.beta = cfg.splicing ? xexp10(th[i++]) : 0.0;
  R.scal = cfg.scaling_column ? th[i++] : (model == 2 ? 0.0 : 1.0);
  R.koff = xexp10(lkoff);
  R.lam = xexp10(llam);
  for (int k = 0; k < S; ++k) {
    R.kon[k] = xexp10(lk[k]);
    R.alp[k] = xexp10(la[k]);
    R.gam[k] = xexp10(lg[k]);
    R.amax[k] = R.alp[k] * xpow(1.0 + (double)(k + 1) / (double)S, R.scal);
  }
  for (int k = S; k < kMaxSteps; ++k) R.kon[k] = R.alp[k] = R.gam[k] = R.amax[k] = 0.0;
  for (int k = 0; k < S; ++k)
    if (!(R.kon[k] < INFINITY) || !(R.alp[k] < INFINITY) || !(R.gam[k] < INFINITY)) return -5;
  if (!(R.koff < INFINITY) || R.lam != R.lam || R.scal != R.scal || R.scal < 0.0) return -5;
  return 0;
}

// ---------------------------------------------------------------------------
// Statistics from per-(condition, age) moments m[(j*A+a)*5 + {mu_u, mu_l,
// var_u, cov_ul, var_l}], in the reference layout
// [pulse_mean A | pulse_ff A | chase_mean A | chase_ff A | ratio J |
//  mean_corr J | corr_mean J].  Sums run left to right.
// ---------------------------------------------------------------------------
ABC_HD double wsum(const double* w, const double* x, int A) {
  double s = w[0] * x[0];
  for (int a = 1; a < A; ++a) s = s + w[a] * x[a];
  return s;
}
// the statistics of condition j (its ratio, mean_corr and corr_mean, and the
// pulse or chase means and Fano factors when j is that condition); conditions
// write disjoint entries, so they may run in any order or in parallel
ABC_HD void stats_from_moments_cond(const DevCfg& cfg, const double* m, const double* age_dist, double* st, int j) {
  const int A = cfg.n_ages, J = cfg.n_conds;
  double w[kMaxAges], mu[kMaxAges], ml[kMaxAges], vu[kMaxAges], cv[kMaxAges], vl[kMaxAges];
  {
    for (int a = 0; a < A; ++a) {
      const double* g = m + (j * A + a) * 5;
      w[a] = age_dist[a * J + j];
      mu[a] = g[0];
      ml[a] = g[1];
      vu[a] = g[2];
      cv[a] = g[3];
      vl[a] = g[4];
    }
    const double swu = wsum(w, mu, A), swl = wsum(w, ml, A);
    st[4 * A + j] = swl / (swu + swl);
    // wcov(mu, mu), wcov(ml, ml) and wcov(mu, ml): the means above and the deviations once
    double suu = 0.0, sll = 0.0, sul = 0.0;
    for (int a = 0; a < A; ++a) {
      const double du = mu[a] - swu, dl = ml[a] - swl;
      const double pu = w[a] * (du * du), pl = w[a] * (dl * dl), pc = w[a] * (du * dl);
      suu = a ? suu + pu : pu;
      sll = a ? sll + pl : pl;
      sul = a ? sul + pc : pc;
    }
    const double tvu = wsum(w, vu, A) + suu;
    const double tvl = wsum(w, vl, A) + sll;
    const double stds = sqrt(fabs(tvu * tvl));
    st[4 * A + J + j] = wsum(w, cv, A) / stds;
    st[4 * A + 2 * J + j] = sul / stds;
    int off = (j == cfg.pulse_stat) ? 0 : (j == cfg.chase_stat) ? 2 * A : -1;
    if (off >= 0) {
      for (int a = 0; a < A; ++a) {
        double tot = mu[a] + ml[a];
        double eps = (tot == 0.0) ? 0.0001 : 0.0;
        st[off + a] = tot;
        st[off + A + a] = ((vu[a] + 2.0 * cv[a]) + vl[a]) / (tot + eps);
      }
      if (off == 0 && j == cfg.chase_stat)  // one condition gives both families
        for (int a = 0; a < 2 * A; ++a) st[2 * A + a] = st[a];
    }
  }
}

// int128 -> double with the oracle's rounding (exact below 2^62).
ABC_HD double i128_to_double(__int128 x) {
  const __int128 lim = ((__int128)1) << 62;
  if (x >= -lim && x <= lim) return (double)(int64_t)x;
  bool neg = x < 0;
  unsigned __int128 ux = neg ? (unsigned __int128)(-x) : (unsigned __int128)x;
  double hi = (double)(uint64_t)(ux >> 64);
  double lo = (double)(uint64_t)ux;
  double v = hi * 18446744073709551616.0 + lo;
  return neg ? -v : v;
}

}  // namespace abc
