// moment_fp32.cu — production mode of the moment-ODE simulation (the FP64
// unit moment.cu is the oracle-exact mode): same exponential midpoint rule on
// the same substep grid, in FP32, with the augmented state ordered
//   [1, E G, Var G, E u, E l, Cov(G,u), Cov(G,l), Var u, Cov(u,l), Var l]
// in which the moment matrix of scripts/model.jl:74-86 is lower triangular:
// every moment depends only on itself and on moments listed before it.
// Products of such matrices keep not only the triangle but the pattern of
// 38 entries that the matrix's dependencies allow (row_mask); the other 17 are
// exact zeros and are neither stored nor multiplied.  Taylor order 8 after scaling
// to a column-sum norm <= 1/2 (truncation < 6e-9, below FP32's 6e-8
// resolution).  Substep and labelling indices are integers (the grid is aligned
// with every breakpoint), so the per-substep work has no FP64 operation; rates,
// times and the statistics stay in FP64.  The transient phase applies the
// one-cycle propagator (the ordered product of the cycle's unlabelled substep
// propagators) once per cycle.  The default substep is cycle / 80 (every pulse,
// chase and age of the reference grid is a multiple of it): against the
// reference's recovered statistics it is as close as cycle / 400, and within
// 3e-3 of it.
//
// Kernels per chunk of particles:
//   rates   a thread per particle;
//   exp     a propagator per thread, its 38 entries in registers.  (A lane per
//           entry of one product at a time, operands in shared memory, took
//           some 60 times as many instructions.)
//   cycle   the one-cycle propagators, a column of a quarter per thread;
//   walk    a thread per particle: the transient, then the unlabelled stretch
//           that the particle's trajectories share, walked once;
//   paths   the labelled and chased rest of the trajectories, a lane per
//           (condition, age);
//   stats   capture and statistics.
// 10,000 particles: 0.56 ms; 14.4 with one CTA per particle doing all of it,
// trajectories from their first substep on.
#include <cuda_runtime.h>

#include <algorithm>

#include "moment.cuh"

namespace abc {
namespace {

constexpr int kTaylor = 8;
constexpr int kNnz = 38, kQuads = 10;  // stored entries of a propagator; 16-byte pieces, the last one half padding
constexpr int kExpThreads = 128;
constexpr int kQuarters = 4;  // parts of the cycle multiplied separately
constexpr int kCycleParticles = 8;
constexpr int kPathParticles = 8;  // a warp of the path kernel: these x kPathGroup pairs, two per lane
constexpr int kPathGroup = 2 * 32 / kPathParticles;
constexpr int kWalkStages = 8, kPathStages = 4;  // substeps whose propagators are on their way

// Scratch of a chunk of n particles.  The particle is the fastest index of the
// propagators: threads of neighbouring particles read and write whole lines.
enum { kRateOn = 0, kRateAlp = kMaxSteps, kRateGam = 2 * kMaxSteps, kRateOff = 3 * kMaxSteps, kRateLam, kRateScal,
       kRateBad, kRates };
struct MomScratch {
  float4* props;  // [labelled][substep][kQuads][n]
  float4* phi;    // [kQuads][n]
  float* start;   // [pairs, in plan order][n][NA]
  float* mom;     // [n][pairs][5]
  float* rates;   // [kRates][n]
  int64_t n;
};

// columns of the stored entries of row r, as bits
__device__ __forceinline__ constexpr unsigned row_mask(int r) {
  return r == 0   ? 0x001u
         : r == 1 ? 0x003u
         : r == 2 ? 0x007u
         : r == 3 ? 0x00bu
         : r == 4 ? 0x013u
         : r == 5 ? 0x027u
         : r == 6 ? 0x047u
         : r == 7 ? 0x0afu
         : r == 8 ? 0x167u
                  : 0x257u;
}
__device__ __forceinline__ bool stored(int r, int c) { return (row_mask(r) >> c) & 1u; }

// position of the entry (r, c) among the stored ones (row by row)
__device__ __forceinline__ int pos_of(int r, int c) {
  constexpr int first[NA] = {0, 1, 3, 6, 9, 12, 16, 20, 26, 32};
  return first[r] + __popc(row_mask(r) & ((1u << c) - 1u));
}

struct Prop {
  float v[4 * kQuads];
};

__device__ __forceinline__ void set_quad(Prop& P, int i, float4 q) {
  P.v[4 * i] = q.x;
  P.v[4 * i + 1] = q.y;
  P.v[4 * i + 2] = q.z;
  P.v[4 * i + 3] = q.w;
}

// src: the first piece, stride apart
__device__ __forceinline__ void load_prop(const float4* src, int64_t stride, Prop& P) {
#pragma unroll
  for (int i = 0; i < kQuads; ++i) set_quad(P, i, src[i * stride]);
}

// y <- P y, each row from its first entry on
__device__ __forceinline__ void apply(const Prop& P, float (&y)[NA]) {
  float z[NA];
  int i = 0;
#pragma unroll
  for (int r = 0; r < NA; ++r) {
    float acc = 0.0f;
#pragma unroll
    for (int c = 0; c < NA; ++c)
      if (stored(r, c)) acc = fmaf(P.v[i++], y[c], acc);
    z[r] = acc;
  }
#pragma unroll
  for (int r = 0; r < NA; ++r) y[r] = z[r];
}

__device__ __forceinline__ void cp_async16(void* dst, const void* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((unsigned)__cvta_generic_to_shared(dst)), "l"(src)
               : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int LEFT>
__device__ __forceinline__ void cp_async_wait() {
  asm volatile("cp.async.wait_group %0;" ::"n"(LEFT) : "memory");
}

// rates of one particle, times the substep
__global__ void moment_rates_kernel(MomArgs a, int64_t p0, MomScratch ws) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x, n = ws.n;
  if (i >= n) return;
  PRec R;
  const bool bad = parse_theta(a.cfg, a.model, a.theta + (p0 + i) * a.ld, R);
  const double h = a.h;
  float* out = ws.rates + i;
  for (int k = 0; k < a.cfg.n_steps; ++k) {
    out[(kRateOn + k) * n] = bad ? 0.0f : (float)(R.kon[k] * h);
    out[(kRateAlp + k) * n] = bad ? 0.0f : (float)(R.alp[k] * h);
    out[(kRateGam + k) * n] = bad ? 0.0f : (float)(R.gam[k] * h);
  }
  out[kRateOff * n] = bad ? 0.0f : (float)(R.koff * h);
  out[kRateLam * n] = bad ? 0.0f : (float)R.lam;
  out[kRateScal * n] = bad ? 0.0f : (float)R.scal;
  out[kRateBad * n] = bad ? 1.0f : 0.0f;
}

// The propagator of one substep of one particle per thread (blockIdx.y: the substep,
// the labelled ones second).  The generator in the permuted order (rows: 0 const,
// 1 EG, 2 VarG, 3 Eu, 4 El, 5 CovGu, 6 CovGl, 7 Varu, 8 Covul, 9 Varl; rates
// already times h):
//   (1,0) kon (1,1) -ks | (2,0) kon (2,1) koff - kon (2,2) -2 ks | (3,1) a1 (3,3) -g |
//   (4,1) a2 (4,4) -g | (5,2) a1 (5,5) -(ks + g) | (6,2) a2 (6,6) -(ks + g) |
//   (7,1) a1 (7,3) g (7,5) 2 a1 (7,7) -2 g | (8,5) a2 (8,6) a1 (8,8) -2 g |
//   (9,1) a2 (9,4) g (9,6) 2 a2 (9,9) -2 g,   ks = kon + koff, a1 = al (1 - lam), a2 = al lam
__global__ void __launch_bounds__(kExpThreads) moment_exp_kernel(MomArgs a, MomScratch ws) {
  const int64_t i = (int64_t)blockIdx.x * kExpThreads + threadIdx.x, n = ws.n;
  if (i >= n) return;
  const int lab = (int)blockIdx.y / a.nsub, idx = (int)blockIdx.y - lab * a.nsub, k = idx / a.per_step;
  const float* m = ws.rates + i;
  const float hf = (float)a.h, invT = (float)(1.0 / a.cfg.cycle);
  const float ph = ((float)idx + 0.5f) * hf;
  // alpha(t) = alpha_k size^s, size = 1 + phase / T (model.jl:25-27)
  const float al = m[(kRateAlp + k) * n] * exp2f(m[kRateScal * n] * __log2f(fmaf(ph, invT, 1.0f)));
  const float lam = lab ? m[kRateLam * n] : 0.0f;
  const float kon = m[(kRateOn + k) * n], koff = m[kRateOff * n], g = m[(kRateGam + k) * n];
  const float ks = kon + koff, a1 = al * (1.0f - lam), a2 = al * lam;
  const float kd = koff - kon, ks2 = -2.0f * ks, kg = -(ks + g), a1d = 2.0f * a1, a2d = 2.0f * a2, g2 = -2.0f * g;
  // column-sum norm
  float norm = (0.0f + fabsf(kon)) + fabsf(kon);
  norm = fmaxf(norm, ((((fabsf(ks) + fabsf(kd)) + fabsf(a1)) + fabsf(a2)) + fabsf(a1)) + fabsf(a2));
  norm = fmaxf(norm, (fabsf(ks2) + fabsf(a1)) + fabsf(a2));
  norm = fmaxf(norm, fabsf(g) + fabsf(g));
  norm = fmaxf(norm, (fabsf(kg) + fabsf(a1d)) + fabsf(a2));
  norm = fmaxf(norm, (fabsf(kg) + fabsf(a1)) + fabsf(a2d));
  norm = fmaxf(norm, fabsf(g2));
  int sq = 0;
  while (norm > 0.5f && sq < 256) {  // (a norm beyond FP32's range ends here too)
    norm *= 0.5f;
    sq++;
  }
  const float sc = ldexpf(1.0f, -sq);
  float A[NA][NA];  // only the entries named below are ever read
  A[1][0] = A[2][0] = kon * sc;
  A[1][1] = -ks * sc;
  A[2][1] = kd * sc;
  A[2][2] = ks2 * sc;
  A[3][1] = A[5][2] = A[7][1] = A[8][6] = a1 * sc;
  A[4][1] = A[6][2] = A[8][5] = A[9][1] = a2 * sc;
  A[3][3] = A[4][4] = -g * sc;
  A[5][5] = A[6][6] = kg * sc;
  A[7][3] = A[9][4] = g * sc;
  A[7][5] = a1d * sc;
  A[9][6] = a2d * sc;
  A[7][7] = A[8][8] = A[9][9] = g2 * sc;
  constexpr unsigned kGen[NA] = {0x000u, 0x003u, 0x007u, 0x00au, 0x012u, 0x024u, 0x044u, 0x0aau, 0x160u, 0x252u};
  // E <- I + A E / q, q = 8 .. 1.  Row r of A E needs rows up to r of E only, so
  // descending rows overwrite in place.
  Prop E;
#pragma unroll
  for (int r = 0; r < NA; ++r)
#pragma unroll
    for (int c = 0; c < NA; ++c)
      if (stored(r, c)) E.v[pos_of(r, c)] = r == c ? 1.0f : 0.0f;
#pragma unroll 1
  for (int q = kTaylor; q >= 1; --q) {
    const float inv = 1.0f / (float)q;
#pragma unroll
    for (int r = NA - 1; r >= 1; --r) {
      float t[NA];
#pragma unroll
      for (int c = 0; c < NA; ++c) {
        if (!stored(r, c)) continue;
        float acc = 0.0f;
#pragma unroll
        for (int j = 0; j < NA; ++j)
          if (((kGen[r] >> j) & 1u) && stored(j, c)) acc = fmaf(A[r][j], E.v[pos_of(j, c)], acc);
        t[c] = fmaf(acc, inv, r == c ? 1.0f : 0.0f);
      }
#pragma unroll
      for (int c = 0; c < NA; ++c)
        if (stored(r, c)) E.v[pos_of(r, c)] = t[c];
    }
  }
  // E <- E E, likewise
#pragma unroll 1
  for (int s = 0; s < sq; ++s) {
#pragma unroll
    for (int r = NA - 1; r >= 0; --r) {
      float t[NA];
#pragma unroll
      for (int c = 0; c < NA; ++c) {
        if (!stored(r, c)) continue;
        float acc = 0.0f;
#pragma unroll
        for (int j = 0; j < NA; ++j)
          if (stored(r, j) && stored(j, c)) acc = fmaf(E.v[pos_of(r, j)], E.v[pos_of(j, c)], acc);
        t[c] = acc;
      }
#pragma unroll
      for (int c = 0; c < NA; ++c)
        if (stored(r, c)) E.v[pos_of(r, c)] = t[c];
    }
  }
  E.v[kNnz] = E.v[kNnz + 1] = 0.0f;
  float4* dst = ws.props + (int64_t)blockIdx.y * kQuads * n + i;
#pragma unroll
  for (int q = 0; q < kQuads; ++q)
    dst[q * n] = make_float4(E.v[4 * q], E.v[4 * q + 1], E.v[4 * q + 2], E.v[4 * q + 3]);
}

// division map (model.jl:98-111) in the permuted order
__device__ __forceinline__ void divide_p(float (&v)[NA]) {
  const float eu = v[3], el = v[4];
  v[5] *= 0.5f;
  v[6] *= 0.5f;
  v[7] = 0.25f * v[7] + 0.25f * eu;
  v[9] = 0.25f * v[9] + 0.25f * el;
  v[8] *= 0.25f;
  v[3] = 0.5f * eu;
  v[4] = 0.5f * el;
}

// original moment index of each permuted position
__device__ __forceinline__ int orig_of(int r) {
  // 0 const, 1 EG(0), 2 VarG(3), 3 Eu(1), 4 El(2), 5 CovGu(4), 6 CovGl(5), 7 Varu(6), 8 Covul(7), 9 Varl(8)
  const int map[NA] = {-1, 0, 3, 1, 2, 4, 5, 6, 7, 8};
  return map[r];
}

// One-cycle propagators without labelling, Phi = P[nsub-1] ... P[0]: the
// columns of each contiguous quarter P[q1-1] ... P[q0], applied from the identity,
// then those of the quarters' product.  Threads: column of quarter x particle.
__global__ void __launch_bounds__(kCycleParticles * kQuarters * NA, 3) moment_cycle_kernel(int nsub, MomScratch ws) {
  __shared__ float sq[kQuarters][4 * kQuads][kCycleParticles];
  const int pi = threadIdx.x % kCycleParticles, w = threadIdx.x / (kCycleParticles * NA);
  const int c = threadIdx.x / kCycleParticles % NA;
  const int64_t i = (int64_t)blockIdx.x * kCycleParticles + pi, n = ws.n;
  float q[NA];
#pragma unroll
  for (int r = 0; r < NA; ++r) q[r] = r == c ? 1.0f : 0.0f;
  if (i < n) {
    const int q1 = (w + 1) * nsub / kQuarters;
#pragma unroll 1
    for (int s = w * nsub / kQuarters; s < q1; ++s) {
      float4 b[kQuads];  // every load under way before the first use
#pragma unroll
      for (int e = 0; e < kQuads; ++e) b[e] = ws.props[((int64_t)s * kQuads + e) * n + i];
      Prop P;
#pragma unroll
      for (int e = 0; e < kQuads; ++e) set_quad(P, e, b[e]);
      apply(P, q);
    }
  }
#pragma unroll
  for (int r = 0; r < NA; ++r)
    if (stored(r, c)) sq[w][pos_of(r, c)][pi] = q[r];
  __syncthreads();
  if (w == 0) {
    for (int v = 1; v < kQuarters; ++v) {
      Prop P;
#pragma unroll
      for (int e = 0; e < kNnz; ++e) P.v[e] = sq[v][e][pi];
      apply(P, q);
    }
#pragma unroll
    for (int r = 0; r < NA; ++r)
      if (stored(r, c)) sq[0][pos_of(r, c)][pi] = q[r];  // read by this column's thread alone until here
    if (c < 4 * kQuads - kNnz) sq[0][kNnz + c][pi] = 0.0f;
  }
  __syncthreads();
  if (w == 0 && i < n)
    ws.phi[c * n + i] = make_float4(sq[0][4 * c][pi], sq[0][4 * c + 1][pi], sq[0][4 * c + 2][pi], sq[0][4 * c + 3][pi]);
}

// Transient phase (model.jl:114-142): one cycle from iv, then cycles until the
// moments of E G, E u, Var G, Cov(G,u), Var u change by <= 1 %; then the
// unlabelled substeps: global substep s (midpoint t0 + (s + 1/2) h), divisions
// at multiples of nsub, the state kept where a pair's labelling starts.  A serial chain
// of some 300 substeps per particle, few warps: each thread copies its
// propagators kWalkStages substeps ahead into shared memory.
__global__ void __launch_bounds__(32) moment_walk_kernel(MomArgs a, int64_t p0, MomScratch ws,
                                                         const __grid_constant__ MomPlan plan) {
  __shared__ float4 ring[kWalkStages][kQuads][32];
  const int64_t i = (int64_t)blockIdx.x * 32 + threadIdx.x, n = ws.n;
  const bool live = i < n && ws.rates[kRateBad * n + (i < n ? i : 0)] == 0.0f;
  const unsigned lanes = __ballot_sync(0xffffffffu, live);
  if (!live) return;
  const int nsub = a.nsub, steps = plan.lo[plan.n - 1];
  auto fetch = [&](int s, int sub) {  // sub = s mod nsub
    if (s < steps)
#pragma unroll
      for (int q = 0; q < kQuads; ++q)
        cp_async16(&ring[s % kWalkStages][q][threadIdx.x], ws.props + ((int64_t)sub * kQuads + q) * n + i);
    cp_async_commit();
  };
  int ahead = 0;
  for (int s = 0; s < kWalkStages - 1; ++s) {
    fetch(s, ahead);
    if (++ahead == nsub) ahead = 0;
  }
  Prop P;
  load_prop(ws.phi + i, n, P);
  float y[NA], e1[NA];
  y[0] = 1.0f;
#pragma unroll
  for (int r = 1; r < NA; ++r) y[r] = (float)a.iv[orig_of(r)];
  apply(P, y);
#pragma unroll
  for (int r = 0; r < NA; ++r) e1[r] = y[r];
  int it = 0;
  bool conv = false;
  while (!conv && it <= 100) {
    it++;
    divide_p(y);
    apply(P, y);
    const int chk[5] = {1, 3, 2, 5, 7};
    int nz = 0, ok = 0;
#pragma unroll
    for (int q = 0; q < 5; ++q) {
      const int r = chk[q];
      if (e1[r] > 0.0f) {
        nz++;
        if (fabsf((e1[r] - y[r]) / e1[r]) <= 0.01f) ok++;
      }
    }
    conv = ok == nz;
#pragma unroll
    for (int r = 0; r < NA; ++r) e1[r] = y[r];
  }
  divide_p(y);
  if (a.iters) a.iters[p0 + i] = it;
  int q = 0, idx = 0;
  for (int s = 0;; ++s) {
    for (; q < plan.n && plan.lo[q] <= s; ++q) {
      float* start = ws.start + ((int64_t)q * n + i) * NA;
#pragma unroll
      for (int r = 0; r < NA; r += 2) *reinterpret_cast<float2*>(start + r) = make_float2(y[r], y[r + 1]);
    }
    if (q == plan.n) break;
    __syncwarp(lanes);  // the slot read last is free
    fetch(s + kWalkStages - 1, ahead);
    if (++ahead == nsub) ahead = 0;
    if (idx == nsub) {
      idx = 0;
      divide_p(y);
    }
    ++idx;
    cp_async_wait<kWalkStages - 1>();  // substep s is there: a thread reads only what it copied
    load_prop(&ring[s % kWalkStages][0][threadIdx.x], 32, P);
    apply(P, y);
  }
}

// Trajectories (model.jl:146-199) from the start of their labelling.  A warp
// holds kPathGroup neighbouring pairs (blockIdx.y) of kPathParticles particles:
// the pairs walk the substeps together, each joining at its lo and leaving at
// its end, so a particle's lanes read the same propagators, which the warp copies
// kPathStages substeps ahead into shared memory.  What bounds it is reading them
// from there (40 cycles of the multiprocessor's load path a substep, FMAs 38), so
// a lane walks two neighbouring pairs on one read (10,000 particles: 226 us with one pair
// per lane and 4 particles per warp, 153 now).  Groups of 8 neighbours by lo
// take 131 steps for 32 of the reference's hourly pairs, groups of 32 take 232.
__global__ void __launch_bounds__(32) moment_path_kernel(MomArgs a, MomScratch ws,
                                                         const __grid_constant__ MomPlan plan) {
  __shared__ float4 ring[kPathStages][2][kQuads][kPathParticles];
  const int JA = plan.n, nsub = a.nsub, lane = threadIdx.x;
  const int64_t n = ws.n;
  const int pi = lane % kPathParticles, slot = (int)blockIdx.y * kPathGroup + lane / kPathParticles * 2;
  const int64_t i = (int64_t)blockIdx.x * kPathParticles + pi;
  const bool good = i < n && ws.rates[kRateBad * n + (i < n ? i : 0)] == 0.0f;
  bool live[2];
  int lo[2], hi[2], end[2];
  unsigned first = 0x7fffffffu, last = 0, un = 0x7fffffffu, la = 0;
  float y[2][NA];
#pragma unroll
  for (int e = 0; e < 2; ++e) {
    live[e] = good && slot + e < JA;
    lo[e] = live[e] ? max(plan.lo[slot + e], 0) : 0x7fffffff;
    end[e] = live[e] ? max(plan.end[slot + e], 0) : 0;
    hi[e] = live[e] ? min(max(plan.hi[slot + e], 0), end[e]) : 0;
    if (live[e]) {
      first = min(first, (unsigned)lo[e]);
      last = max(last, (unsigned)end[e]);
      un = min(un, (unsigned)hi[e]);
      la = max(la, (unsigned)hi[e]);
    }
#pragma unroll
    for (int r = 0; r < NA; ++r) y[e][r] = live[e] ? ws.start[((int64_t)(slot + e) * n + i) * NA + r] : 0.0f;
  }
  // substeps s0 .. s1 of the warp; the unlabelled propagators serve from un on, the labelled ones up to la
  // (without a valid particle in the warp `first` is the largest int, beyond which nothing may be counted: s0 = s1 = 0)
  const int s1 = (int)__reduce_max_sync(0xffffffffu, last), s0 = min((int)__reduce_min_sync(0xffffffffu, first), s1);
  un = __reduce_min_sync(0xffffffffu, un);
  la = __reduce_max_sync(0xffffffffu, la);
  const int64_t src0 = lane / kPathParticles * n + min(i, n - 1);
  auto fetch = [&](int s, int sub) {
#pragma unroll
    for (int lab = 0; lab < 2; ++lab) {
      if (s >= s1 || (lab ? s >= (int)la : s < (int)un)) continue;
      const float4* src = ws.props + (int64_t)(lab * nsub + sub) * kQuads * n + src0;
      float4* dst = &ring[s % kPathStages][lab][0][0] + lane;
#pragma unroll
      for (int q = 0; q < kQuads * kPathParticles; q += 32)
        if (q + lane < kQuads * kPathParticles) cp_async16(dst + q, src + q / kPathParticles * n);
    }
    cp_async_commit();
  };
  int idx = s0 % nsub, ahead = idx;
  for (int t = 0; t < kPathStages - 1; ++t) {
    fetch(s0 + t, ahead);
    if (++ahead == nsub) ahead = 0;
  }
  for (int s = s0; s < s1; ++s) {
    cp_async_wait<kPathStages - 2>();
    __syncwarp();  // every lane's pieces of substep s are there, and the slot read last is free
    fetch(s + kPathStages - 1, ahead);
    if (++ahead == nsub) ahead = 0;
    const bool on0 = s >= lo[0] && s < end[0], on1 = s >= lo[1] && s < end[1];
    const bool lab0 = s < hi[0], lab1 = s < hi[1];
    if (on0 || on1) {
      const float4(*src)[kQuads][kPathParticles] = ring[s % kPathStages];
      Prop P;
      load_prop(&src[(on0 ? lab0 : lab1) ? 1 : 0][0][pi], kPathParticles, P);
      if (on0) {
        if (idx == 0 && s > 0) divide_p(y[0]);
        apply(P, y[0]);
      }
      if (on1) {
        if (on0 && lab0 != lab1) load_prop(&src[lab1 ? 1 : 0][0][pi], kPathParticles, P);
        if (idx == 0 && s > 0) divide_p(y[1]);
        apply(P, y[1]);
      }
    }
    if (++idx == nsub) idx = 0;
  }
#pragma unroll
  for (int e = 0; e < 2; ++e) {
    if (!live[e]) continue;
    float* mo = ws.mom + ((int64_t)i * JA + plan.pair[slot + e]) * 5;
    mo[0] = y[e][3];
    mo[1] = y[e][4];
    mo[2] = y[e][7];
    mo[3] = y[e][8];
    mo[4] = y[e][9];
  }
}

}  // namespace

size_t moment_f32_scratch(int64_t P, int nsub, int pairs) {
  const size_t n = (size_t)moment_chunk(P, nsub, kQuads * sizeof(float4));
  return n * ((2 * (size_t)nsub + 1) * kQuads * sizeof(float4) + ((size_t)pairs * (NA + 5) + kRates) * sizeof(float));
}

cudaError_t launch_moment_f32(const MomArgs& a, cudaStream_t s) {
  if (a.P <= 0) return cudaSuccess;
  const MomPlan plan = moment_plan(a);
  const int pairs = plan.n;
  const int64_t chunk = moment_chunk(a.P, a.nsub, kQuads * sizeof(float4));
  for (int64_t p0 = 0; p0 < a.P; p0 += chunk) {
    const int64_t n = std::min<int64_t>(chunk, a.P - p0);
    MomScratch ws;
    ws.n = n;
    ws.props = reinterpret_cast<float4*>(a.scratch);
    ws.phi = ws.props + (size_t)n * 2 * a.nsub * kQuads;
    ws.start = reinterpret_cast<float*>(ws.phi + (size_t)n * kQuads);
    ws.mom = ws.start + (size_t)n * pairs * NA;
    ws.rates = ws.mom + (size_t)n * pairs * 5;
    moment_rates_kernel<<<(unsigned)((n + 31) / 32), 32, 0, s>>>(a, p0, ws);
    moment_exp_kernel<<<dim3((unsigned)((n + kExpThreads - 1) / kExpThreads), 2 * a.nsub), kExpThreads, 0, s>>>(a, ws);
    moment_cycle_kernel<<<(unsigned)((n + kCycleParticles - 1) / kCycleParticles), kCycleParticles * kQuarters * NA, 0,
                          s>>>(a.nsub, ws);
    moment_walk_kernel<<<(unsigned)((n + 31) / 32), 32, 0, s>>>(a, p0, ws, plan);
    moment_path_kernel<<<dim3((unsigned)((n + kPathParticles - 1) / kPathParticles),
                              (pairs + kPathGroup - 1) / kPathGroup), 32, 0, s>>>(a, ws, plan);
    moment_stats_kernel<float><<<(unsigned)((n + kStatParticles - 1) / kStatParticles), 128, stat_smem(pairs), s>>>(
        a, p0, n, ws.mom, ws.rates + kRateBad * n);
    const cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return e;
  }
  return cudaSuccess;
}

}  // namespace abc
