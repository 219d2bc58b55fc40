// moment.cu — the reference's deterministic simulation on the GPU: the
// 9-moment linear ODE of the telegraph model with labelling (scripts/model.jl:
// 67-96), its periodic steady state (transient_phase, :114-142), the
// multi-cycle trajectories with division (:98-111, :146-199), the capture
// moment transform (downsample, :221-239) and the 53 statistics
// (scripts/abc_simulation.jl:13-62).
//
// y' = A(t) y + b(t) is integrated by the exponential midpoint rule on a grid
// of step h aligned with every breakpoint: each substep applies
// expm(h A(t_mid)) to the state augmented with a constant 1.  The 10 x 10
// exponentials come from scaling and squaring with an 18-term Taylor
// polynomial in Horner form.  Every sum runs in the order of the FP64 C oracle
// (built with -fmad=false here and -ffp-contract=off there), so the results are
// bit-identical.  What is left out of the sums adds an exact zero: the generator has 24
// nonzero entries, and its powers keep to the 38 that the moments'
// dependencies allow (row_mask).
//
// Kernels per chunk of particles, all bound by the FP64 pipe (or, for few
// particles, by its latency):
//   rates   a thread per particle;
//   exp     a propagator per thread, its entries in registers;
//   walk    the transient phase, then the unlabelled stretch that a particle's
//           trajectories share, walked once: a serial chain, so a lane per row
//           of the state, three particles per warp;
//   paths   the labelled and chased rest of the trajectories, a lane per
//           (condition, age);
//   stats   capture and statistics (moment.cuh).
// 500 particles on the default grid (400 substeps a cycle): 17 ms; 144 with one CTA
// per particle, full 10 x 10 products by lanes over shared memory, and every trajectory
// walked from its first substep on.  One particle: 3.6 and 42 ms.
#include <cuda_runtime.h>

#include "distance.cuh"
#include "moment.cuh"

namespace abc {
namespace {

constexpr int kNnz = 38;
constexpr int kTaylor = 18;
constexpr int kExpThreads = 128;
constexpr int kWalkGroup = 3;  // particles per warp of the walk
constexpr int kPathParticles = 4, kPathGroup = 32 / kPathParticles;  // a warp of the path kernel

enum { kRateOn = 0, kRateAlp = kMaxSteps, kRateGam = 2 * kMaxSteps, kRateOff = 3 * kMaxSteps, kRateLam, kRateScal,
       kRateBad, kRates };
// Scratch of a chunk of n particles, the particle the fastest index of the propagators
struct MomScratch {
  double* props;  // [labelled][substep][kNnz][n]
  double* start;  // [pairs, in plan order][n][NA]
  double* mom;    // [n][pairs][5]
  double* rates;  // [kRates][n]
  int64_t n;
};

// State order: 0 E G, 1 E u, 2 E l, 3 Var G, 4 Cov(G,u), 5 Cov(G,l), 6 Var u,
// 7 Cov(u,l), 8 Var l, 9 the constant 1.  Columns of row r of a propagator and
// of the generator, as bits.
__device__ __forceinline__ constexpr unsigned row_mask(int r) {
  return r == 0   ? 0x201u
         : r == 1 ? 0x203u
         : r == 2 ? 0x205u
         : r == 3 ? 0x209u
         : r == 4 ? 0x219u
         : r == 5 ? 0x229u
         : r == 6 ? 0x25bu
         : r == 7 ? 0x2b9u
         : r == 8 ? 0x32du
                  : 0x200u;
}
__device__ __forceinline__ constexpr unsigned gen_mask(int r) {
  return r == 0   ? 0x201u
         : r == 1 ? 0x003u
         : r == 2 ? 0x005u
         : r == 3 ? 0x209u
         : r == 4 ? 0x018u
         : r == 5 ? 0x028u
         : r == 6 ? 0x053u
         : r == 7 ? 0x0b0u
         : r == 8 ? 0x125u
                  : 0x000u;
}
// the rows so that each comes before the ones that it depends on
__device__ __forceinline__ constexpr int row_at(int i) {
  return i == 0 ? 8 : i == 1 ? 7 : i == 2 ? 6 : i == 3 ? 5 : i == 4 ? 4 : i == 5 ? 2 : i == 6 ? 1 : i == 7 ? 3 : i == 8 ? 0 : 9;
}
__device__ __forceinline__ bool stored(int r, int c) { return (row_mask(r) >> c) & 1u; }
// position of the first stored entry of row r, and of the entry (r, c) (row by row)
__device__ __forceinline__ constexpr int first_of(int r) {
  return r == 0   ? 0
         : r == 1 ? 2
         : r == 2 ? 5
         : r == 3 ? 8
         : r == 4 ? 11
         : r == 5 ? 15
         : r == 6 ? 19
         : r == 7 ? 25
         : r == 8 ? 31
                  : 37;
}
__device__ __forceinline__ int pos_of(int r, int c) { return first_of(r) + __popc(row_mask(r) & ((1u << c) - 1u)); }

__global__ void moment_rates_kernel(MomArgs a, int64_t p0, MomScratch ws) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x, n = ws.n;
  if (i >= n) return;
  PRec R;
  const bool bad = parse_theta(a.cfg, a.model, a.theta + (p0 + i) * a.ld, R);
  double* out = ws.rates + i;
  for (int k = 0; k < a.cfg.n_steps; ++k) {
    out[(kRateOn + k) * n] = bad ? 0.0 : R.kon[k];
    out[(kRateAlp + k) * n] = bad ? 0.0 : R.alp[k];
    out[(kRateGam + k) * n] = bad ? 0.0 : R.gam[k];
  }
  out[kRateOff * n] = bad ? 0.0 : R.koff;
  out[kRateLam * n] = bad ? 0.0 : R.lam;
  out[kRateScal * n] = bad ? 0.0 : R.scal;
  out[kRateBad * n] = bad ? 1.0 : 0.0;
}

// t / d for a small whole d, y = RN(1 / d)
__device__ __forceinline__ double div_whole(double t, double d, double y) {
  return (__double_as_longlong(t) << 1) == 0 ? t : div_rn(t, d, y);
}

// The propagator of one substep of one particle per thread (blockIdx.y: the
// substep, the labelled ones second): expm of the generator times h (rows of
// A(t), model.jl:74-86) by scaling to a column-sum norm <= 1/2, the Taylor sum in
// Horner form and squaring back.
__global__ void __launch_bounds__(kExpThreads) moment_exp_kernel(MomArgs a, MomScratch ws) {
  const int64_t i = (int64_t)blockIdx.x * kExpThreads + threadIdx.x, n = ws.n;
  if (i >= n || ws.rates[kRateBad * n + i] != 0.0) return;
  const int lab = (int)blockIdx.y / a.nsub, idx = (int)blockIdx.y - lab * a.nsub, k = idx / a.per_step;
  const double* m = ws.rates + i;
  const double h = a.h;
  const double ph = ((double)idx + 0.5) * h;
  const double al = m[(kRateAlp + k) * n] * xpow(1.0 + ph / a.cfg.cycle, m[kRateScal * n]);
  const double kon = m[(kRateOn + k) * n], koff = m[kRateOff * n], gam = m[(kRateGam + k) * n];
  const double lam = lab ? m[kRateLam * n] : 0.0;
  const double ks = kon + koff;
  double Ai = kon * h, Aks = -ks * h, Akd = (koff - kon) * h, Ak2 = (-2.0 * ks) * h, Akg = -(ks + gam) * h;
  double Aa1 = ((1.0 - lam) * al) * h, Aa2 = (lam * al) * h, Ag = gam * h;
  // (2 x a1 and the like are exact multiples of these)
  double norm = ((((fabs(Aks) + fabs(Aa1)) + fabs(Aa2)) + fabs(Akd)) + fabs(Aa1)) + fabs(Aa2);  // E G
  norm = fmax(norm, fabs(Ag) + fabs(Ag));                                                       // E u, E l
  norm = fmax(norm, (fabs(Ak2) + fabs(Aa1)) + fabs(Aa2));                                       // Var G
  norm = fmax(norm, (fabs(Akg) + fabs(2.0 * Aa1)) + fabs(Aa2));                                 // Cov(G,u)
  norm = fmax(norm, (fabs(Akg) + fabs(Aa1)) + fabs(2.0 * Aa2));                                 // Cov(G,l)
  norm = fmax(norm, fabs(Ai) + fabs(Ai));                                                       // 1
  int sq = 0;
  while (norm > 0.5 && sq < 2048) {  // (an infinite norm ends here too)
    norm *= 0.5;
    sq++;
  }
  const double sc = ldexp(1.0, -sq);
  Ai *= sc; Aks *= sc; Akd *= sc; Ak2 *= sc; Akg *= sc; Aa1 *= sc; Aa2 *= sc; Ag *= sc;
  double A[NA][NA];  // only the entries named below are ever read
  A[0][0] = Aks; A[0][9] = Ai;
  A[1][0] = Aa1; A[1][1] = -Ag;
  A[2][0] = Aa2; A[2][2] = -Ag;
  A[3][0] = Akd; A[3][3] = Ak2; A[3][9] = Ai;
  A[4][3] = Aa1; A[4][4] = Akg;
  A[5][3] = Aa2; A[5][5] = Akg;
  A[6][0] = Aa1; A[6][1] = Ag; A[6][4] = 2.0 * Aa1; A[6][6] = -2.0 * Ag;
  A[7][4] = Aa2; A[7][5] = Aa1; A[7][7] = -2.0 * Ag;
  A[8][0] = Aa2; A[8][2] = Ag; A[8][5] = 2.0 * Aa2; A[8][8] = -2.0 * Ag;
  double E[kNnz];
#pragma unroll
  for (int r = 0; r < NA; ++r)
#pragma unroll
    for (int c = 0; c < NA; ++c)
      if (stored(r, c)) E[pos_of(r, c)] = r == c ? 1.0 : 0.0;
  // E <- A E / q + I; a row of A E needs E's rows only up to itself (row_at), so it is overwritten in place
#pragma unroll 1
  for (int q = kTaylor; q >= 1; --q) {
    const double qd = (double)q, y = 1.0 / qd;
#pragma unroll
    for (int ri = 0; ri < NA - 1; ++ri) {
      const int r = row_at(ri);
      double t[NA];
#pragma unroll
      for (int c = 0; c < NA; ++c) {
        if (!stored(r, c)) continue;
        bool open = false;
        double s = 0.0;
#pragma unroll
        for (int j = 0; j < NA; ++j)
          if (((gen_mask(r) >> j) & 1u) && stored(j, c)) {
            const double x = A[r][j] * E[pos_of(j, c)];
            s = open ? s + x : x;
            open = true;
          }
        t[c] = div_whole(s, qd, y);
        if (r == c) t[c] = t[c] + 1.0;
      }
#pragma unroll
      for (int c = 0; c < NA; ++c)
        if (stored(r, c)) E[pos_of(r, c)] = t[c];
    }
  }
#pragma unroll 1
  for (int s2 = 0; s2 < sq; ++s2) {
#pragma unroll
    for (int ri = 0; ri < NA - 1; ++ri) {
      const int r = row_at(ri);
      double t[NA];
#pragma unroll
      for (int c = 0; c < NA; ++c) {
        if (!stored(r, c)) continue;
        bool open = false;
        double s = 0.0;
#pragma unroll
        for (int j = 0; j < NA; ++j)
          if (stored(r, j) && stored(j, c)) {
            const double x = E[pos_of(r, j)] * E[pos_of(j, c)];
            s = open ? s + x : x;
            open = true;
          }
        t[c] = s;
      }
#pragma unroll
      for (int c = 0; c < NA; ++c)
        if (stored(r, c)) E[pos_of(r, c)] = t[c];
    }
  }
  double* dst = ws.props + (int64_t)blockIdx.y * kNnz * n + i;
#pragma unroll
  for (int e = 0; e < kNnz; ++e) dst[e * n] = E[e];
}

// division map (periodic_boundary, model.jl:98-111); halves and quarters are exact
__device__ __forceinline__ void divide(double (&v)[NA]) {
  const double e1 = v[1], e2 = v[2];
  v[4] = v[4] * 0.5;
  v[5] = v[5] * 0.5;
  v[6] = v[6] * 0.25 + e1 * 0.25;
  v[8] = v[8] * 0.25 + e2 * 0.25;
  v[7] = v[7] * 0.25;
  v[1] = e1 * 0.5;
  v[2] = e2 * 0.5;
}

// the same when lane base + r holds v[r]
__device__ __forceinline__ double divide_lane(double v, int r, int base) {
  const double e1 = __shfl_sync(0xffffffffu, v, base + 1), e2 = __shfl_sync(0xffffffffu, v, base + 2);
  const double half = v * 0.5, quarter = v * 0.25;
  const double sum = quarter + (r == 6 ? e1 : e2) * 0.25;
  return r == 1 || r == 2 || r == 4 || r == 5 ? half : r == 7 ? quarter : r == 6 || r == 8 ? sum : v;
}

// Transient phase (model.jl:114-142): one cycle from iv, then cycles until the
// moments of E G, E u, Var G, Cov(G,u), Var u change by <= 1 %; then the
// unlabelled substeps from t0 on, the state kept where a pair's labelling starts.
// Lane 10 p + r holds row r of the state of the warp's particle p; the
// next substep's entries are loaded while one is applied.
__global__ void __launch_bounds__(32) moment_walk_kernel(MomArgs a, int64_t p0, MomScratch ws,
                                                         const __grid_constant__ MomPlan plan) {
  constexpr int kRow = 6;  // entries of the longest row
  const int64_t n = ws.n;
  const int lane = threadIdx.x, grp = min(lane / NA, kWalkGroup - 1), r = min(lane - grp * NA, NA - 1);
  const int base = grp * NA;
  const int64_t i = (int64_t)blockIdx.x * kWalkGroup + grp, ic = min(i, n - 1);
  const bool live = lane < kWalkGroup * NA && i < n && ws.rates[kRateBad * n + ic] == 0.0;
  // (an invalid particle beside a valid one has no propagators: its lanes feed only each other)
  if (!__any_sync(0xffffffffu, live)) return;
  const int nsub = a.nsub;
  int col[kRow], len = 0;
#pragma unroll
  for (int c = 0; c < NA; ++c)
    if ((row_mask(r) >> c) & 1u) {
#pragma unroll
      for (int e = 0; e < kRow; ++e)
        if (e == len) col[e] = c;
      ++len;
    }
#pragma unroll
  for (int e = 0; e < kRow; ++e)
    if (e >= len) col[e] = 0;
  const double* P0 = ws.props + (int64_t)first_of(r) * n + ic;
  double nxt[kRow];
  auto load = [&](int sub) {
#pragma unroll
    for (int e = 0; e < kRow; ++e) nxt[e] = e < len ? P0[((int64_t)sub * kNnz + e) * n] : 0.0;
  };
  // y <- P y with the entries loaded last, those of substep `then` loaded meanwhile
  auto step = [&](double y, int then) {
    double cur[kRow];
#pragma unroll
    for (int e = 0; e < kRow; ++e) cur[e] = nxt[e];
    load(then);
    double s = 0.0;
#pragma unroll
    for (int e = 0; e < kRow; ++e) {
      const double x = cur[e] * __shfl_sync(0xffffffffu, y, base + col[e]);
      s = e == 0 ? x : e < len ? s + x : s;
    }
    return s;
  };
  auto cycle = [&](double y) {
    for (int s = 0; s < nsub; ++s) y = step(y, s + 1 == nsub ? 0 : s + 1);
    return y;
  };
  load(0);
  const unsigned particle = 0x3ffu << base;
  double e1 = cycle(r < 9 ? a.iv[r] : 1.0), e2 = e1;
  int it = 0;
  bool conv = !live;
  while (__any_sync(0xffffffffu, !conv)) {
    const double y = cycle(divide_lane(e1, r, base));
    const bool chk = r == 0 || r == 1 || r == 3 || r == 4 || r == 6;
    const bool nzl = chk && e1 > 0.0;
    const bool okl = nzl && fabs((e1 - y) / e1) <= 0.01;
    const unsigned ok = __ballot_sync(0xffffffffu, okl) & particle, nz = __ballot_sync(0xffffffffu, nzl) & particle;
    if (!conv) {
      it++;
      e2 = y;
      conv = __popc(ok) == __popc(nz) || it > 100;
      e1 = y;
    }
  }
  if (live && r == 0 && a.iters) a.iters[p0 + i] = it;
  double y = divide_lane(e2, r, base);
  int q = 0, idx = 0;
  for (int s = 0;; ++s) {
    for (; q < plan.n && plan.lo[q] <= s; ++q)
      if (live) ws.start[((int64_t)q * n + i) * NA + r] = y;
    if (q == plan.n) break;
    if (idx == nsub) {
      idx = 0;
      y = divide_lane(y, r, base);
    }
    ++idx;
    y = step(y, idx == nsub ? 0 : idx);
  }
}

// Trajectories (model.jl:146-199) from the start of their labelling.  A warp
// holds kPathGroup neighbouring pairs (blockIdx.y) of kPathParticles particles;
// the pairs walk the substeps together, each joining at its lo and leaving at
// its end.
__global__ void __launch_bounds__(32) moment_path_kernel(MomArgs a, MomScratch ws,
                                                         const __grid_constant__ MomPlan plan) {
  const int JA = plan.n, nsub = a.nsub, lane = threadIdx.x;
  const int64_t n = ws.n;
  const int slot = (int)blockIdx.y * kPathGroup + lane / kPathParticles;
  const int64_t i = (int64_t)blockIdx.x * kPathParticles + lane % kPathParticles;
  const bool live = i < n && slot < JA && ws.rates[kRateBad * n + (i < n ? i : 0)] == 0.0;
  const int lo = live ? max(plan.lo[slot], 0) : 0x7fffffff, end = live ? max(plan.end[slot], 0) : 0;
  const int hi = live ? plan.hi[slot] : 0;
  const int s0 = (int)__reduce_min_sync(0xffffffffu, (unsigned)lo);
  const int s1 = (int)__reduce_max_sync(0xffffffffu, (unsigned)end);
  if (!live) return;
  double y[NA];
#pragma unroll
  for (int r = 0; r < NA; ++r) y[r] = ws.start[((int64_t)slot * n + i) * NA + r];
  int idx = s0 % nsub;
  for (int s = s0; s < s1; ++s) {
    if (s >= lo && s < end) {
      if (idx == 0 && s > 0) divide(y);
      const double* P = ws.props + (int64_t)((s < hi ? nsub : 0) + idx) * kNnz * n + i;
      double z[NA];
      int e = 0;
#pragma unroll
      for (int r = 0; r < NA; ++r) {
        double acc = 0.0;
        bool open = false;
#pragma unroll
        for (int c = 0; c < NA; ++c)
          if (stored(r, c)) {
            const double x = P[e++ * n] * y[c];
            acc = open ? acc + x : x;
            open = true;
          }
        z[r] = acc;
      }
#pragma unroll
      for (int r = 0; r < NA; ++r) y[r] = z[r];
    }
    if (++idx == nsub) idx = 0;
  }
  double* mo = ws.mom + ((int64_t)i * JA + plan.pair[slot]) * 5;
  mo[0] = y[1];
  mo[1] = y[2];
  mo[2] = y[6];
  mo[3] = y[7];
  mo[4] = y[8];
}

}  // namespace

size_t moment_f64_scratch(int64_t P, int nsub, int pairs) {
  const size_t n = (size_t)moment_chunk(P, nsub, kNnz * sizeof(double));
  return n * ((size_t)2 * nsub * kNnz + (size_t)pairs * (NA + 5) + kRates) * sizeof(double);
}

cudaError_t launch_moment(const MomArgs& a, cudaStream_t s) {
  if (a.P <= 0) return cudaSuccess;
  const MomPlan plan = moment_plan(a);
  const int pairs = plan.n;
  const int64_t chunk = moment_chunk(a.P, a.nsub, kNnz * sizeof(double));
  for (int64_t p0 = 0; p0 < a.P; p0 += chunk) {
    const int64_t n = std::min<int64_t>(chunk, a.P - p0);
    MomScratch ws;
    ws.n = n;
    ws.props = reinterpret_cast<double*>(a.scratch);
    ws.start = ws.props + (size_t)n * 2 * a.nsub * kNnz;
    ws.mom = ws.start + (size_t)n * pairs * NA;
    ws.rates = ws.mom + (size_t)n * pairs * 5;
    moment_rates_kernel<<<(unsigned)((n + 31) / 32), 32, 0, s>>>(a, p0, ws);
    moment_exp_kernel<<<dim3((unsigned)((n + kExpThreads - 1) / kExpThreads), 2 * a.nsub), kExpThreads, 0, s>>>(a, ws);
    moment_walk_kernel<<<(unsigned)((n + kWalkGroup - 1) / kWalkGroup), 32, 0, s>>>(a, p0, ws, plan);
    moment_path_kernel<<<dim3((unsigned)((n + kPathParticles - 1) / kPathParticles),
                              (pairs + kPathGroup - 1) / kPathGroup), 32, 0, s>>>(a, ws, plan);
    moment_stats_kernel<double><<<(unsigned)((n + kStatParticles - 1) / kStatParticles), 128, stat_smem(pairs), s>>>(
        a, p0, n, ws.mom, ws.rates + kRateBad * n);
    const cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return e;
  }
  return cudaSuccess;
}

}  // namespace abc
