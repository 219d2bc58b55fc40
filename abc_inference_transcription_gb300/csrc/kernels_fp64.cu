// kernels_fp64.cu — prior draw, particle setup, FP64 (oracle-mode) SSA and the
// fused capture + statistics kernel.  Built with -fmad=false: every FP64
// result here is bit-identical to the FP64 CPU oracle.
#include <type_traits>

#include "kernels.h"
#include "sampler32.cuh"

namespace abc {

// ---------------------------------------------------------------------------
// Prior draw (fix_params, scripts/abc_simulation.jl:3-11): one thread per
// particle, Philox stream ST_PRIOR, cell 0.  Column order of theta:
// kon(1|S), koff, alpha(1|S), gamma(1|S), lambda, [beta], [scaling].
// ---------------------------------------------------------------------------
__global__ void prior_kernel(PriorArgs A) {
  int64_t p = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (p >= A.n_particles) return;
  Rng r;
  rng_init(r, A.seed, ST_PRIOR, 0u, (uint32_t)(A.p_offset + p));
  double* th = A.theta + p * A.cfg.npar;
  const int S = A.cfg.n_steps;
  int i = 0;
  uint32_t a, b;
  for (int rate = 0; rate < 4; ++rate) {
    const double lo = A.lo[rate], hi = A.hi[rate];
    bool varies = (A.model == 3 && rate == 0) || (A.model == 4 && rate == 2) || (A.model == 5 && rate == 3);
    rng_pair(r, a, b);
    double base = lo + (hi - lo) * u52(a, b);
    if (!varies) {
      th[i++] = base;
    } else if (A.vary_mode == 0) {
      th[i++] = base;
      for (int k = 1; k < S; ++k) {
        rng_pair(r, a, b);
        th[i++] = lo + (hi - lo) * u52(a, b);
      }
    } else {
      for (int k = 0; k < S; ++k) {
        rng_pair(r, a, b);
        th[i++] = base + (A.lf0 + (A.lf1 - A.lf0) * u52(a, b));
      }
    }
  }
  rng_pair(r, a, b);
  th[i++] = A.lo[4] + (A.hi[4] - A.lo[4]) * u52(a, b);
  if (A.cfg.splicing) {
    rng_pair(r, a, b);
    th[i++] = A.lo[5] + (A.hi[5] - A.lo[5]) * u52(a, b);
  }
  if (A.cfg.scaling_column) {
    rng_pair(r, a, b);
    th[i++] = xexp10(A.lo[6] + (A.hi[6] - A.lo[6]) * u52(a, b));
  }
}

cudaError_t launch_prior(const PriorArgs& a, cudaStream_t s) {
  if (a.n_particles <= 0) return cudaSuccess;
  int blocks = (int)((a.n_particles + 127) / 128);
  prior_kernel<<<blocks, 128, 0, s>>>(a);
  return cudaGetLastError();
}

// ---------------------------------------------------------------------------
// theta -> rates, thinning bounds and initial state, LANES lanes per particle
// (model.cuh has the formulas; every operation and its order are the
// oracle's, so the record is bit-identical).  One thread per particle ran
// six dependent passes over a cycle's 80 sub-steps, 0.69 ms for one particle
// and for 10,000 alike.  Here lane k holds age step k, the sub-steps' rates and
// sources are computed side by side, and only the recurrences stay serial, two
// operations each, the passes from different start values on different lanes.
// Bound by the FP64 pipe, which a warp's instruction holds whatever the
// number of lanes with work: 8 lanes per particle, so that the serial parts
// occupy it once for four particles, or 32 while the particles' warps do not fill the
// GPU.  One particle: 107 us with 8 lanes and sources inside the recurrences, 73 now; 10,000:
// 455 us, 342 now.
// ---------------------------------------------------------------------------
constexpr int kSetupLanes = 8;  // 32 up to a warp per scheduler
static_assert(kSetupLanes >= kMaxSteps, "lane k holds age step k");
constexpr int kMaxSub = kMaxSteps * kIcSub;

struct SetupShared {
  PRec R;
  double ginf[kMaxSteps], eG[kMaxSteps], phG[kMaxSteps], em[kMaxSteps], phm[kMaxSteps];
  double ec[kMaxSteps], phc[kMaxSteps], ev[kMaxSteps], phv[kMaxSteps];
  double g[kMaxSub];  // E G at the start of each sub-step, then 2 alpha
  double aG[kMaxSub], sm[kMaxSub], sc[kMaxSub];  // alpha E G, sources of E u and Cov(G, u)
  double x[4][kMaxSub + 1];  // E u from 0 and from 1, Cov from 0 and from 1, at the sub-steps' ends
  double w2[kMaxSub];        // sources of Var u (those of two starts overwrite sm and sc)
};

// The periodic moments by the particle's lanes; lane 0 writes the record
template <int LANES>
__device__ void initial_moments_lanes(const DevCfg& cfg, SetupShared& W, int r) {
  const int S = cfg.n_steps, N = S * kIcSub;
  const double T = cfg.cycle;
  const double h = (T / (double)S) / (double)kIcSub;
  if (r < S) {
    const double kG = W.R.kon[r] + W.R.koff, gam = W.R.gam[r];
    W.ginf[r] = W.R.kon[r] / kG;
    phi_pair(kG * h, W.eG[r], W.phG[r]);
    phi_pair(gam * h, W.em[r], W.phm[r]);
    phi_pair((kG + gam) * h, W.ec[r], W.phc[r]);
    phi_pair((2.0 * gam) * h, W.ev[r], W.phv[r]);
  }
  __syncwarp();
  // E G over one cycle from 0 (even lanes) and from 1 (odd lanes): its fixed point
  double g = (double)(r & 1);
  for (int k = 0; k < S; ++k) {
    const double gi = W.ginf[k], eG = W.eG[k];
    for (int i = 0; i < kIcSub; ++i) g = gi + (g - gi) * eG;
  }
  const double z0 = __shfl_sync(0xffffffffu, g, 0, LANES), e0 = __shfl_sync(0xffffffffu, g, 1, LANES);
  double g0 = z0 / (1.0 - (e0 - z0));
  if (!(g0 > 0.0)) g0 = 0.0;
  if (g0 > 1.0) g0 = 1.0;
  g = g0;
  for (int k = 0; k < S; ++k) {
    const double gi = W.ginf[k], eG = W.eG[k];
    for (int i = 0; i < kIcSub; ++i) {
      if (r == 0) W.g[k * kIcSub + i] = g;
      g = gi + (g - gi) * eG;
    }
  }
  __syncwarp();
  for (int q = r; q < N; q += LANES) {
    const int k = q / kIcSub;
    const double ph = ((double)q + 0.5) * h;
    const double a = W.R.alp[k] * xpow(1.0 + ph / T, W.R.scal);
    const double gi = W.ginf[k];
    const double Gavg = gi + (W.g[q] - gi) * W.phG[k];
    W.sm[q] = ((a * Gavg) * h) * W.phm[k];
    W.sc[q] = ((a * (Gavg * (1.0 - Gavg))) * h) * W.phc[k];
    W.aG[q] = a * Gavg;
    W.g[q] = 2.0 * a;
  }
  __syncwarp();
  // the cycle map of (E u, Cov, Var u) from 0, (1, 0, 0), (0, 1, 0), (0, 0, 1): E u and
  // Cov depend on their own start alone (lanes 0..3 of x), the sources of Var u
  // on both, for three pairs of starts, and Var u is a recurrence on them
  const unsigned F = 0xffffffffu;
  {
    double y = (double)(r & 1);
    const double* E = (r & 2) ? W.ec : W.em;
    const double* s = (r & 2) ? W.sc : W.sm;
    if (r < 4) W.x[r][0] = y;
    for (int k = 0; k < S; ++k) {
      const double ek = E[k];
      for (int i = 0; i < kIcSub; ++i) {
        const int q = k * kIcSub + i;
        y = y * ek + s[q];
        if (r < 4) W.x[r][q + 1] = y;
      }
    }
  }
  __syncwarp();
  for (int item = r; item < 3 * N; item += LANES) {
    const int start = item / N, q = item - start * N, k = q / kIcSub;
    const double* m = W.x[start == 1 ? 1 : 0];
    const double* c = W.x[start == 2 ? 3 : 2];
    const double src = (W.aG[q] + W.R.gam[k] * (0.5 * (m[q] + m[q + 1]))) + W.g[q] * (0.5 * (c[q] + c[q + 1]));
    (start == 0 ? W.sm : start == 1 ? W.sc : W.w2)[q] = (src * h) * W.phv[k];
  }
  __syncwarp();
  double v = r == 3 ? 1.0 : 0.0;
  {
    const double* w = r == 1 ? W.sc : r == 2 ? W.w2 : W.sm;
    for (int k = 0; k < S; ++k) {
      const double ev = W.ev[k];
      for (int i = 0; i < kIcSub; ++i) v = v * ev + w[k * kIcSub + i];
    }
  }
  double m = W.x[r == 1 ? 1 : 0][N], c = W.x[r == 2 ? 3 : 2][N];
  v = v * 0.25 + m * 0.25;
  m = m * 0.5;
  c = c * 0.5;
  const double b1 = __shfl_sync(F, m, 0, LANES), b2 = __shfl_sync(F, c, 0, LANES);
  const double b3 = __shfl_sync(F, v, 0, LANES);
  const double mmm = __shfl_sync(F, m, 1, LANES) - b1, mvm = __shfl_sync(F, v, 1, LANES) - b3;
  const double mcc = __shfl_sync(F, c, 2, LANES) - b2, mvc = __shfl_sync(F, v, 2, LANES) - b3;
  const double mvv = __shfl_sync(F, v, 3, LANES) - b3;
  double m0 = b1 / (1.0 - mmm);
  double c0 = b2 / (1.0 - mcc);
  double v0 = ((b3 + mvm * m0) + mvc * c0) / (1.0 - mvv);
  if (!(m0 > 0.0)) m0 = 0.0;
  if (!(v0 > 0.0)) v0 = 0.0;
  if (!(c0 == c0)) c0 = 0.0;
  if (r == 0) {
    W.R.g0 = g0;
    W.R.u0 = m0;
    W.R.s0 = 0.0;
    W.R.c0 = c0;
    W.R.v0 = v0;
  }
}

// initial_means (model.cuh), splicing models: the four passes on lanes 0..3
template <int LANES>
__device__ void initial_means_lanes(const DevCfg& cfg, SetupShared& W, int r) {
  double x0 = r == 1 ? 1.0 : 0.0, x1 = r == 2 ? 1.0 : 0.0, x2 = r == 3 ? 1.0 : 0.0;
  if (r < 4) mean_cycle(cfg, W.R, x0, x1, x2);
  const unsigned F = 0xffffffffu;
  double b[3], col[3][3];
  b[0] = __shfl_sync(F, x0, 0, LANES);
  b[1] = __shfl_sync(F, x1, 0, LANES);
  b[2] = __shfl_sync(F, x2, 0, LANES);
  for (int i = 0; i < 3; ++i) {
    col[i][0] = __shfl_sync(F, x0, i + 1, LANES);
    col[i][1] = __shfl_sync(F, x1, i + 1, LANES);
    col[i][2] = __shfl_sync(F, x2, i + 1, LANES);
  }
  if (r == 0) solve_initial_means(cfg, b, col, W.R);
}

template <int LANES>
__global__ void __launch_bounds__(32) setup_kernel(SetupArgs A) {
  constexpr int kSetupParticles = 32 / LANES;  // per block (one warp)
  __shared__ SetupShared sh[kSetupParticles];
  const int r = threadIdx.x % LANES, slot = threadIdx.x / LANES;
  const int64_t p = (int64_t)blockIdx.x * kSetupParticles + slot;
  const bool here = p < A.n_particles;
  const DevCfg& cfg = A.cfg;
  const int S = cfg.n_steps;
  SetupShared& W = sh[slot];
  PRec& R = W.R;
  const int model = !here ? 0 : A.models ? A.models[p] : A.model;
  bool bad = !(model >= 1 && model <= 5);
  // rates: lane k takes age step k; columns hcat(kon, koff, alpha, gamma, lambda, [beta], [scaling]),
  // the model's varying rate expanded over the steps
  if (!bad) {
    const double* th = A.theta + p * A.ld_theta;
    const int nk = model == 3 ? S : 1, na = model == 4 ? S : 1, ng = model == 5 ? S : 1;
    const int ikoff = nk, ia = nk + 1, ig = ia + na, il = ig + ng;
    int i = il + 1;
    const double beta = cfg.splicing ? xexp10(th[i++]) : 0.0;
    const double scal = cfg.scaling_column ? th[i++] : (model == 2 ? 0.0 : 1.0);
    const double koff = xexp10(th[ikoff]), lam = xexp10(th[il]);
    double kon = 0.0, alp = 0.0, gam = 0.0, amax = 0.0;
    if (r < S) {
      kon = xexp10(th[nk > 1 ? r : 0]);
      alp = xexp10(th[ia + (na > 1 ? r : 0)]);
      gam = xexp10(th[ig + (ng > 1 ? r : 0)]);
      amax = alp * xpow(1.0 + (double)(r + 1) / (double)S, scal);
      bad = !(kon < INFINITY) || !(alp < INFINITY) || !(gam < INFINITY);
    }
    bad = bad || !(koff < INFINITY) || lam != lam || scal != scal || scal < 0.0;
    if (r < kMaxSteps) {
      R.kon[r] = kon;
      R.alp[r] = alp;
      R.gam[r] = gam;
      R.amax[r] = amax;
    }
    if (r == 0) {
      R.koff = koff;
      R.lam = lam;
      R.beta = beta;
      R.scal = scal;
    }
  }
  const unsigned mine = (0xffffffffu >> (32 - LANES)) << (slot * LANES);
  bad = (__ballot_sync(0xffffffffu, bad) & mine) != 0u;
  if (bad) {
    // a harmless record: the trajectory sees no reactions
    if (r < kMaxSteps) R.kon[r] = R.alp[r] = R.gam[r] = R.amax[r] = 0.0;
    if (r == 0) {
      R.koff = R.lam = R.beta = R.scal = R.g0 = R.u0 = R.s0 = R.c0 = R.v0 = 0.0;
      R.cost = 1.0;
      if (here) atomicOr(A.status, STF_NONFINITE);
    }
  } else if (r == 0) {
    R.c0 = R.v0 = 0.0;
  }
  __syncwarp();
  // (the lanes of a bad record run along, for the shuffles, and are not kept)
  PRec keep = {};
  if (bad && r == 0) keep = R;
  if (cfg.splicing)
    initial_means_lanes<LANES>(cfg, W, r);
  else
    initial_moments_lanes<LANES>(cfg, W, r);
  // work estimate: switching + transcription + decay events over the horizon
  double rate = 0.0, mine_k = 0.0;
  if (r < S) {
    const double pon = R.kon[r] / (R.kon[r] + R.koff);
    mine_k = 2.0 * pon * R.koff + 2.0 * pon * R.amax[r];
  }
  for (int k = 0; k < S; ++k) rate = rate + __shfl_sync(0xffffffffu, mine_k, k, LANES);
  if (r == 0) {
    if (bad)
      R = keep;
    else
      R.cost = (double)(cfg.ages[0] - cfg.t0) * rate / (double)S + 1.0;
  }
  __syncwarp();
  if (!here) return;
  const double* src = reinterpret_cast<const double*>(&R);
  double* dst = reinterpret_cast<double*>(&A.rec[p]);
  for (int i = r; i < (int)(sizeof(PRec) / sizeof(double)); i += LANES) dst[i] = src[i];
  // rates in log2 units (times log2 e), so the production kernel's waiting
  // time is -log2(U) / a0 without a conversion per event
  constexpr double kL2E = 1.4426950408889634;
  const int rk = r < kMaxSteps ? r : kMaxSteps - 1;
  float kon = (float)(R.kon[rk] * kL2E), alp = (float)(R.alp[rk] * kL2E), gam = (float)(R.gam[rk] * kL2E);
  float amax = (float)(R.amax[rk] * kL2E), koff = (float)(R.koff * kL2E), beta = (float)(R.beta * kL2E);
  float lam = (float)R.lam, scal = (float)R.scal;
  if (A.fp32) {
    // rates beyond the FP32 range would stall the production kernel's clock
    const bool ok = koff < 1e30f && beta < 1e30f && kon < 1e30f && alp < 1e30f && gam < 1e30f;
    if ((__ballot_sync(mine, !ok) & mine) != 0u) {
      if (r == 0) atomicOr(A.status, STF_NONFINITE);
      kon = alp = gam = amax = koff = lam = beta = scal = 0.0f;
    }
  }
  PRecF& F = A.recf[p];
  if (r < kMaxSteps) {
    F.kon[r] = kon;
    F.alp[r] = alp;
    F.gam[r] = gam;
    F.amax[r] = amax;
  }
  if (r == 0) {
    F.koff = koff;
    F.lam = lam;
    F.beta = beta;
    F.scal = scal;
  }
}

cudaError_t launch_setup(const SetupArgs& a, cudaStream_t s) {
  if (a.n_particles <= 0) return cudaSuccess;
  if (a.n_particles <= 4 * (int64_t)a.sms) {
    setup_kernel<32><<<(unsigned)a.n_particles, 32, 0, s>>>(a);
  } else {
    constexpr int per = 32 / kSetupLanes;
    setup_kernel<kSetupLanes><<<(unsigned)((a.n_particles + per - 1) / per), 32, 0, s>>>(a);
  }
  return cudaGetLastError();
}

// ---------------------------------------------------------------------------
// SSA, FP64 oracle mode.
// ---------------------------------------------------------------------------
// Persistent: every lane owns one trajectory at a time and pulls the next
// (particle, cell) item from the global counter (warp-aggregated atomics).
__global__ void __launch_bounds__(128) ssa_kernel_fp64(SsaArgs A) {
  const unsigned FULL = 0xffffffffu;
  const int lane = threadIdx.x & 31;
  const int64_t cap = A.cfg.event_cap > 0 ? A.cfg.event_cap : kDefaultEventCap;
  Traj s;
  bool active = false, done = false;
  unsigned long long tot_ev = 0, tot_rej = 0;
  int err = 0;
  while (true) {
    const bool need = !active && !done;
    const unsigned mask = __ballot_sync(FULL, need);
    if (mask) {
      const int leader = __ffs(mask) - 1;
      unsigned long long base = 0;
      if (lane == leader) base = atomicAdd(A.counter, (unsigned long long)__popc(mask));
      base = __shfl_sync(FULL, base, leader);
      if (need) {
        const unsigned long long item = base + (unsigned long long)__popc(mask & ((1u << lane) - 1u));
        if (item >= (unsigned long long)A.n_items) {
          done = true;
        } else {
          traj_init(s, A, (int64_t)item);
          active = true;
        }
      }
    }
    if (__all_sync(FULL, done)) break;
    if (active) {
      const PRec& R = A.rec[s.plocal];
#pragma unroll 1
      for (int it = 0; it < kQuantum; ++it) {
        uint32_t ch;
        bool fin = step_fp64(s, R, A.cfg, ch);
        if (ch == CH_REJ) {
          tot_rej++;
        } else if (ch != CH_NULL) {
          s.ev++;
          if (s.ev > cap) {
            err |= STF_EVENT_CAP;
            fin = true;
          }
        }
        if (s.uu >= kOverflowCount || s.lu >= kOverflowCount || s.us >= kOverflowCount ||
            s.ls >= kOverflowCount) {
          err |= STF_OVERFLOW;
          fin = true;
        }
        if (s.stall > kMaxStall) {
          err |= STF_NONFINITE;
          fin = true;
        }
        if (fin) {
          A.counts[s.out] = make_int2(s.uu + s.us, s.lu + s.ls);
          if (A.events) A.events[s.out] = s.ev;
          if (A.hash) A.hash[s.out] = s.hash;
          tot_ev += (unsigned long long)s.ev;
          active = false;
          break;
        }
      }
    }
  }
  // warp totals -> one atomic per warp
  for (int o = 16; o > 0; o >>= 1) {
    tot_ev += __shfl_xor_sync(FULL, tot_ev, o);
    tot_rej += __shfl_xor_sync(FULL, tot_rej, o);
    err |= __shfl_xor_sync(FULL, err, o);
  }
  if (lane == 0) {
    atomicAdd(&A.totals[0], tot_ev);
    atomicAdd(&A.totals[1], tot_rej);
    if (err) atomicOr(A.status, err);
  }
}

cudaError_t launch_ssa_fp64(const SsaArgs& a, int grid, cudaStream_t s) {
  ssa_kernel_fp64<<<grid, 128, 0, s>>>(a);
  return cudaGetLastError();
}

// One thread per trajectory of the production mode: the gene state from the
// first word of the trajectory's main stream and the moment-matched first
// mRNA count (auxiliary stream), drawn from the distribution traj_init uses
// in the FP64 mode with FP32 samplers.  Runs at full occupancy instead of
// inside the production kernel's divergent refill path.
__global__ void __launch_bounds__(256) init_state_kernel(SsaArgs A) {
  const int64_t P = A.n_items / A.n_cells;
  const int C = (int)A.n_cells;
  __shared__ float mom[5];  // the particle's g0, u0, c0, v0 in FP32, and the rounded mean count
  for (int64_t pl = blockIdx.x; pl < P; pl += gridDim.x) {  // a block per particle, a thread per cell
    if (threadIdx.x == 0) {  // the FP64 -> FP32 conversions once per particle, not per cell
      const PRec& R = A.rec[pl];
      mom[0] = (float)R.g0;
      mom[1] = (float)R.u0;
      mom[2] = (float)R.c0;
      mom[3] = (float)R.v0;
      mom[4] = (float)fmin(floor(R.u0 + 0.5), 1.0e9);  // far above the count limit (2^23), reported there
    }
    __syncthreads();
    const float g0 = mom[0], u0 = mom[1], c0 = mom[2], v0 = mom[3], ur = mom[4];
    const uint32_t particle = (uint32_t)(A.p_offset + pl);
    for (int ci = threadIdx.x; ci < C; ci += blockDim.x) {
      const uint32_t cell = A.cell_id[ci];
      Rng r;
      rng_init(r, A.seed, ST_SSA, cell, particle);
      uint32_t w0, w1;
      rng_pair(r, w0, w1);
      const int G = u24(w0) < g0 ? 1 : 0;
      int u;
      if (A.cfg.splicing) {
        u = (int)ur;
      } else {
        Rng aux;
        rng_init(aux, A.seed, ST_AUX, cell, particle);
        u = initial_count32(g0, u0, c0, v0, G, w1, aux);
      }
      A.counts[pl * A.n_cells + ci] = make_int2(u, G);
    }
    __syncthreads();  // mom is rewritten for the next particle
  }
}

cudaError_t launch_init_states(const SsaArgs& a, int sms, cudaStream_t s) {
  if (a.n_items <= 0 || a.n_cells <= 0) return cudaSuccess;
  const int64_t P = a.n_items / a.n_cells, cap = (int64_t)sms * 16;
  init_state_kernel<<<(unsigned)(P < cap ? P : cap), 256, 0, s>>>(a);
  return cudaGetLastError();
}

// ---------------------------------------------------------------------------
// Capture + statistics: one CTA (8 warps) per particle.  Warp w handles the
// (condition, age) groups w, w+8, ...: each lane thins its cells' counts
// binomially with the cell's capture efficiency (downsample,
// scripts/model.jl:221-239, realised per cell), accumulates exact integer
// moment sums, and the warp reduces them with shuffles.  One thread then
// forms the 4A + 3J statistics (abc_simulation.jl:23-46).
// ---------------------------------------------------------------------------
__device__ __forceinline__ long long shfl_xor_ll(long long v, int o) {
  return __shfl_xor_sync(0xffffffffu, v, o);
}
__device__ __forceinline__ __int128 shfl_xor_i128(__int128 v, int o) {
  unsigned long long lo = (unsigned long long)(unsigned __int128)v;
  long long hi = (long long)(v >> 64);
  lo = __shfl_xor_sync(0xffffffffu, lo, o);
  hi = __shfl_xor_sync(0xffffffffu, hi, o);
  return (__int128)(((unsigned __int128)(unsigned long long)hi << 64) | (unsigned __int128)lo);
}

// NARROW: 64-bit sums of the squared counts (production mode: counts at most
// 2^24, where FP32 increments stop, and at most 2^14 cells per group, so the
// sums stay below 2^62); 128-bit otherwise.
// THREADS: 256, or 1,024 where the launch has too few particles to fill the
// GPU, at most one per SM (the groups are then the parallelism: a particle alone with 55 groups
// of 36 cells takes 90 us in 8 warps, 51 in 32).
template <bool CAP32, bool NARROW, int THREADS>
__global__ void __launch_bounds__(THREADS) stats_kernel(StatsArgs A) {
  __shared__ double mom[kMaxAges * kMaxConds * 5];
  __shared__ double wts[kMaxAges * kMaxConds];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int ng = A.cfg.n_ages * A.cfg.n_conds;
  const int K = 4 * A.cfg.n_ages + 3 * A.cfg.n_conds;
  for (int i = threadIdx.x; i < ng; i += blockDim.x) wts[i] = A.age_dist[i];
  for (int64_t p = blockIdx.x; p < A.n_particles; p += gridDim.x) {
    const int2* cnt = A.counts + p * A.n_cells;
    const uint32_t pg = (uint32_t)(A.p_offset + p);
    for (int g = warp; g < ng; g += (blockDim.x >> 5)) {
      const int g0 = A.gstart[g], g1 = A.gstart[g + 1];
      using Sq = typename std::conditional<NARROW, long long, __int128>::type;
      long long su = 0, sl = 0;
      Sq suu = 0, sll = 0, sul = 0;
      for (int i = g0 + lane; i < g1; i += 32) {
        int2 c = cnt[i];
        Rng r;
        rng_init(r, A.seed, ST_CAPTURE, A.cell_id[i], pg);
        long long cu, cl;
        if (CAP32) {  // FP32 efficiencies: no FP64-pipe work per cell
          const float b32 = A.beta32[i];
          cu = binomial32(r, c.x, b32);
          cl = binomial32(r, c.y, b32);
        } else {
          cu = binomial(r, c.x, A.beta[i]);
          cl = binomial(r, c.y, A.beta[i]);
        }
        if (A.captured) A.captured[p * A.n_cells + i] = make_int2((int)cu, (int)cl);
        su += cu;
        sl += cl;
        suu += (Sq)(cu * cu);
        sll += (Sq)(cl * cl);
        sul += (Sq)(cu * cl);
      }
      for (int o = 16; o > 0; o >>= 1) {
        su += shfl_xor_ll(su, o);
        sl += shfl_xor_ll(sl, o);
        if (NARROW) {
          suu += (Sq)shfl_xor_ll((long long)suu, o);
          sll += (Sq)shfl_xor_ll((long long)sll, o);
          sul += (Sq)shfl_xor_ll((long long)sul, o);
        } else {
          suu += (Sq)shfl_xor_i128((__int128)suu, o);
          sll += (Sq)shfl_xor_i128((__int128)sll, o);
          sul += (Sq)shfl_xor_i128((__int128)sul, o);
        }
      }
      if (lane < 5) {  // lane j forms moment j: [E u, E l, Var u, Cov ul, Var l], one FP64 division each
        const long long n = g1 - g0;
        const double nd = (double)n;
        const double dn = nd * (double)(n - 1);
        __int128 x;
        if (lane == 0) x = su;
        else if (lane == 1) x = sl;
        else if (lane == 2) x = (__int128)n * suu - (__int128)su * su;
        else if (lane == 3) x = (__int128)n * sul - (__int128)su * sl;
        else x = (__int128)n * sll - (__int128)sl * sl;
        mom[g * 5 + lane] = i128_to_double(x) / (lane < 2 ? nd : dn);
      }
    }
    __syncthreads();
    if (warp == 0)  // one condition per lane
      for (int j = lane; j < A.cfg.n_conds; j += 32) stats_from_moments_cond(A.cfg, mom, wts, A.stats + p * K, j);
    __syncthreads();
  }
}

cudaError_t launch_stats(const StatsArgs& a, cudaStream_t s) {
  if (a.n_particles <= 0) return cudaSuccess;
  int blocks = (int)(a.n_particles < 1048576 ? a.n_particles : 1048576);
  if (a.fp32 && a.max_group_cells <= 16384 && blocks <= a.sms)
    stats_kernel<true, true, 1024><<<blocks, 1024, 0, s>>>(a);
  else if (a.fp32 && a.max_group_cells <= 16384)
    stats_kernel<true, true, 256><<<blocks, 256, 0, s>>>(a);
  else if (a.fp32)
    stats_kernel<true, false, 256><<<blocks, 256, 0, s>>>(a);
  else
    stats_kernel<false, false, 256><<<blocks, 256, 0, s>>>(a);
  return cudaGetLastError();
}

int ssa_blocks_per_sm_fp64() {
  int n = 0;
  cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, ssa_kernel_fp64, 128, 0);
  return n;
}

}  // namespace abc
