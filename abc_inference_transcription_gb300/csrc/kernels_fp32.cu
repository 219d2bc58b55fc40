// kernels_fp32.cu — production SSA launch: FP32 propensities, waiting times
// and channel selection with fast intrinsics; compensated FP32 interval clock
// re-anchored at every breakpoint (integer breakpoint grid, or FP64 when the
// configuration's times are not on one).  Built with FMA contraction on.
#include "kernels.h"
#include "ssa_fp32.cuh"

namespace abc {

// Kernel variants the autotuner chooses from: register allocation for 8 or
// 10 resident blocks of 128 threads per SM.
static const int kVariantMinBlocks[kSsaVariants] = {8, 10};

template <bool SPLICE, bool GRID, bool GENSCAL>
static cudaError_t launch_variant(const SsaArgs& b, int variant, int grid, cudaStream_t s) {
  if (variant == 1)
    ssa_kernel_f32<SPLICE, 10, GRID, GENSCAL><<<grid, 128, 0, s>>>(b);
  else
    ssa_kernel_f32<SPLICE, 8, GRID, GENSCAL><<<grid, 128, 0, s>>>(b);
  return cudaGetLastError();
}

template <bool SPLICE, bool GRID>
static cudaError_t launch_scal(const SsaArgs& b, int variant, int grid, cudaStream_t s) {
  // a scaling column in theta gives each particle its own size exponent;
  // without one the exponent is 0 or 1 and the rate is linear in time
  return b.cfg.scaling_column ? launch_variant<SPLICE, GRID, true>(b, variant, grid, s)
                              : launch_variant<SPLICE, GRID, false>(b, variant, grid, s);
}

cudaError_t launch_ssa_fp32(const SsaArgs& a, int grid, cudaStream_t s, int variant) {
  SsaArgs b = a;
  uint32_t k0 = (uint32_t)a.seed, k1 = (uint32_t)(a.seed >> 32);
  for (int r = 0; r < 10; ++r) {
    b.rk[2 * r] = k0;
    b.rk[2 * r + 1] = k1;
    k0 += 0x9E3779B9u;
    k1 += 0xBB67AE85u;
  }
  // integer breakpoints when the configuration's times lie on a power-of-two grid
  if (a.cfg.grid_ok)
    return a.cfg.splicing ? launch_scal<true, true>(b, variant, grid, s) : launch_scal<false, true>(b, variant, grid, s);
  return a.cfg.splicing ? launch_scal<true, false>(b, variant, grid, s) : launch_scal<false, false>(b, variant, grid, s);
}

int ssa_blocks_per_sm_fp32(int variant) {
  int n = 0;
  if (variant == 1)
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, ssa_kernel_f32<false, 10, true, false>, 128, 0);
  else
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, ssa_kernel_f32<false, 8, true, false>, 128, 0);
  return n > 0 ? n : kVariantMinBlocks[variant < 0 || variant >= kSsaVariants ? 0 : variant];
}

// ---------------------------------------------------------------------------
// Work order: particles by expected fired events per trajectory, heaviest
// first (longest-processing-time-first), so the long trajectories start early
// and the end of the persistent kernel is filled with short ones.  64 buckets
// on log2(cost), counting sort; order inside a bucket is arbitrary (it only
// affects scheduling, never results: random streams are keyed by particle).
// ---------------------------------------------------------------------------
__device__ __forceinline__ int cost_bucket(double cost) {
  const int e = (int)((__double_as_longlong(cost) >> 52) & 0x7ff) - 1023;
  const int b = e < 0 ? 0 : (e > 63 ? 63 : e);
  return 63 - b;
}

__global__ void order_hist_kernel(const PRec* rec, int64_t P, unsigned int* hist, WorkPlan* plan) {
  float most = 0.0f;
  unsigned long long sum = 0;
  for (int64_t p = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; p < P; p += (int64_t)gridDim.x * blockDim.x) {
    const double cost = rec[p].cost;
    atomicAdd(&hist[cost_bucket(cost)], 1u);
    const float c = fminf(fmaxf((float)cost, 1.0f), 1e15f);  // NaN counts as 1
    most = fmaxf(most, c);
    sum += (unsigned long long)c;
  }
  for (int o = 16; o > 0; o >>= 1) {
    most = fmaxf(most, __shfl_xor_sync(0xffffffffu, most, o));
    sum += __shfl_xor_sync(0xffffffffu, sum, o);
  }
  if ((threadIdx.x & 31) == 0) {
    atomicMax(&plan->max_cost, __float_as_uint(most));
    atomicAdd(&plan->sum_cost, sum);
  }
}

// Blocks per SM that run.  The resident blocks share a warp's schedulers, so
// a trajectory advances the slower the more of them there are, while the
// total rate saturates.  Measured nanoseconds per iteration of a lane with
// 1..8 blocks of 128 threads per SM: 76, 106, 155, 205, 251, 294, 340, 389
// for a particle of 62,000 iterations per trajectory (236 to 398 x 10^9
// iterations/s over the GPU; alone), 143 to 584 for one of 3,300, whose
// breakpoints weigh more (sum: the mean of the two).  A batch ends no earlier
// than its longest trajectory nor than its sum at the total rate; the number
// of blocks is taken for which the later of the two, plus a quarter of the
// other for the unfilled end, is earliest.  Milliseconds of the SSA kernel on
// five-model prior draws with 1, 2, 3, 4, 8 blocks: 101 particles x 1,437
// cells 15, 17, 25, 27, 25; 2,000 x 2,000 (one block not measured) 74, 69, 76, 80; 10,000 x
// 2,000 396, 360, 352, 363.  Blocks beyond the number leave at once.
// The tables are those of the two-species kernel with a size exponent of 0 or 1 on the
// integer grid.  The other kernels' iterations are longer, by much the same factor in
// every row, which the choice does not depend on.  Milliseconds of the SSA kernel by this
// rule / with all blocks, 2,000 cells, one model's prior draws, 64, 250 and 1,000 particles:
// this kernel 13.9 / 29.0, 18.2 / 29.8, 43.0 / 45.3; splicing 21.3 / 35.2, 27.5 / 42.1,
// 63.1 / 71.7; general exponent 21.4 / 33.1, 25.9 / 41.8, 59.0 / 66.9; both 45.1 / 56.8,
// 46.4 / 83.0, 76.1 / 96.0.  Within 4 % of each other at 4 and 16 particles and at 4,000.
__device__ __forceinline__ int planned_blocks(const WorkPlan* plan, int64_t n_cells, int sms, int most) {
  const float alone[8] = {76.f, 106.f, 155.f, 205.f, 251.f, 294.f, 340.f, 389.f};
  const float sum[8] = {110.f, 148.f, 201.f, 264.f, 319.f, 374.f, 433.f, 487.f};
  const float longest = __uint_as_float(plan->max_cost);
  const float total = (float)plan->sum_cost * (float)n_cells / (float)(128 * sms);
  int best = most;
  float t_best = INFINITY;
  for (int n = 1; n <= 8 && n <= most; ++n) {
    const float a = longest * alone[n - 1], b = total * sum[n - 1] / (float)n;
    const float t = fmaxf(a, b) + 0.25f * fminf(a, b);
    if (t < t_best) {
      t_best = t;
      best = n == 8 ? most : n;
    }
  }
  return best;
}

// hist and cursor of the counting sort; thread 0 also fixes the blocks per SM
// of the production kernel, at most `most`
__global__ void order_scatter_kernel(const PRec* rec, int64_t P, const unsigned int* hist, unsigned int* cursor,
                                     uint32_t* order, WorkPlan* plan, int64_t n_cells, int sms, int most) {
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    const int n = planned_blocks(plan, n_cells, sms, most);
    plan->blocks = n < most ? (unsigned)(n * sms) : 0xffffffffu;
  }
  __shared__ unsigned int start[64];
  if (threadIdx.x == 0) {
    unsigned int run = 0;
    for (int b = 0; b < 64; ++b) {
      start[b] = run;
      run += hist[b];
    }
  }
  __syncthreads();
  for (int64_t p = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; p < P; p += (int64_t)gridDim.x * blockDim.x) {
    const int b = cost_bucket(rec[p].cost);
    order[start[b] + atomicAdd(&cursor[b], 1u)] = (uint32_t)p;
  }
}

cudaError_t launch_work_order(const PRec* rec, int64_t P, unsigned int* scratch, uint32_t* order, int64_t n_cells,
                              int sms, int blocks_per_sm, cudaStream_t s) {
  if (P <= 0) return cudaSuccess;
  WorkPlan* plan = reinterpret_cast<WorkPlan*>(scratch);
  unsigned int* hist128 = scratch + kOrderHist;
  cudaError_t e = cudaMemsetAsync(scratch, 0, kOrderWords * sizeof(unsigned int), s);
  if (e) return e;
  const int blocks = (int)((P + 255) / 256 < 4096 ? (P + 255) / 256 : 4096);
  order_hist_kernel<<<blocks, 256, 0, s>>>(rec, P, hist128, plan);
  order_scatter_kernel<<<blocks, 256, 0, s>>>(rec, P, hist128, hist128 + 64, order, plan, n_cells, sms, blocks_per_sm);
  return cudaGetLastError();
}

}  // namespace abc
