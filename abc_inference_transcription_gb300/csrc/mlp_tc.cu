// mlp_tc.cu — the surrogate's GEMMs on the tcgen05 tensor cores:
//   C[M][N] = sum_k A[m][k] B[n][k]   (both operands K-major, BF16, FP32
//   accumulation in tensor memory), one output tile of 128 x 128 per CTA,
//   ensemble member = blockIdx.z, optional split of the reduction
//   (blockIdx.y = m tile + split * m tiles) for the weight gradients.
// Warp 0 issues TMA loads (3D maps: reduction, rows, member; 64-wide BF16 boxes
// with the 128-byte swizzle) into a 3-stage ring; one lane of warp 1 issues
// tcgen05.mma.kind::f16 (M = N = 128, K = 16); all eight warps then read their 32
// accumulator rows x 64 columns with tcgen05.ld and apply the fused epilogue (bias +
// SiLU, bias, one partial sum per reduction split, or the SiLU derivative), writing the
// row-major result and, where the backward pass needs it, the transposed
// BF16 copy.  Waits are bounded (about one second); a wait that runs out sets
// the error word, and the CTA drains its copies and MMAs before it frees its
// tensor memory.
#include <cuda.h>
#include <cudaTypedefs.h>
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <atomic>
#include <cstring>

#include "kernels.h"
#include "smem_attr.h"
#include "mlp.cuh"
#include "mlp_tc.cuh"
#include "tcgen05.cuh"

namespace abc {
namespace tc {

bool make_map3(CUtensorMap* map, const __nv_bfloat16* base, int64_t K, int64_t ld, int64_t rows, int64_t members,
               int64_t member_stride) {
  static PFN_cuTensorMapEncodeTiled_v12000 encode = nullptr;
  if (!encode) {
    void* fn = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &fn, 12000, cudaEnableDefault, &q) !=
            cudaSuccess ||
        q != cudaDriverEntryPointSuccess || !fn)
      return false;
    encode = (PFN_cuTensorMapEncodeTiled_v12000)fn;
  }
  memset(map, 0, sizeof(*map));
  const int64_t row_bytes = ld * 2;
  int64_t mstride = member_stride * 2;
  if (members <= 1) mstride = ((rows * row_bytes + 15) / 16) * 16;
  cuuint64_t dims[3] = {(cuuint64_t)K, (cuuint64_t)rows, (cuuint64_t)(members < 1 ? 1 : members)};
  cuuint64_t strides[2] = {(cuuint64_t)row_bytes, (cuuint64_t)mstride};
  cuuint32_t box[3] = {(cuuint32_t)kTcBK, 128, 1};
  cuuint32_t estr[3] = {1, 1, 1};
  return encode(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, (void*)base, dims, strides, box, estr,
                CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

}  // namespace tc

namespace {

using namespace tc;

constexpr int BM = 128, BN = 128, BK = kTcBK;
constexpr int kStages = 3;
constexpr uint32_t kTileBytes = BM * BK * 2;  // A and B tiles alike (BN = BM)
constexpr uint32_t kStageBytes = 2 * kTileBytes;
constexpr uint32_t kTmemCols = 128;
constexpr int kSmem = 1024 + kStages * kStageBytes + 128;
constexpr int kThreads = 256;
static_assert(kThreads / 32 * kChunk * kRowF * 4 <= kStages * kStageBytes, "the stages hold the warps' chunks");
// also the transposed copy, whose accesses are whole columns as the lanes stand
__device__ __forceinline__ void store_rows_bf16(float* sm, const float (&x)[kChunk], __nv_bfloat16* base, int64_t ld,
                                                __nv_bfloat16* baseT, int64_t ldT, int rows, int cols, int lane) {
  uint32_t* sw = reinterpret_cast<uint32_t*>(sm);
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    __nv_bfloat16 h[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) h[j] = __float2bfloat16(x[8 * q + j]);
    uint4 pk;
    memcpy(&pk, h, 16);
    *(uint4*)(sw + lane * kRowH + 4 * q) = pk;
    if (baseT && 8 * q < cols && lane < rows) {
#pragma unroll
      for (int j = 0; j < 8; ++j) baseT[(int64_t)(8 * q + j) * ldT + lane] = h[j];
    }
  }
  __syncwarp();
  const int r = lane / 4, c = lane % 4 * 8;
#pragma unroll
  for (int t = 0; t < 4; ++t)
    if (8 * t + r < rows && c < cols)
      *(uint4*)(base + (8 * t + r) * ld + c) = *(const uint4*)(sw + (8 * t + r) * kRowH + c / 2);
  __syncwarp();
}

// one output tile: tile (mt + split * m tiles, nt) of member z
template <int EPI>
__device__ __forceinline__ void gemm_tile(const CUtensorMap& tmA, const CUtensorMap& tmB, const TcGemm& g, int my, int nt,
                                          int z) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = smem_raw + ((1024u - (su32(smem_raw) & 1023u)) & 1023u);
  uint64_t* full = (uint64_t*)(smem + kStages * kStageBytes);
  uint64_t* empty = full + kStages;
  uint64_t* done = empty + kStages;
  uint32_t* tslot = (uint32_t*)(done + 1);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int n_mt = (g.M + BM - 1) / BM;
  const int mt = my % n_mt, split = my / n_mt;
  const int m0 = mt * BM, n0 = nt * BN;
  const int nk = (g.K + BK - 1) / BK;
  const int per = (nk + g.k_split - 1) / g.k_split;
  const int c0 = split * per, c1 = min(nk, c0 + per);
  if (threadIdx.x == 0) {
    for (int st = 0; st < kStages; ++st) {
      mbar_init(&full[st], 1);
      mbar_init(&empty[st], 1);
    }
    mbar_init(done, 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(su32(tslot)),
                 "r"(kTmemCols)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tbase = *tslot;
  const uint32_t sbase = su32(smem);
  const bool work = c1 > c0;
  if (work && warp == 0 && lane == 0) {
    // ---- TMA producer
    int last_par[kStages] = {-1, -1, -1};
    for (int c = c0; c < c1; ++c) {
      const int i = c - c0, st = i % kStages;
      const uint32_t ph = (uint32_t)(i / kStages) & 1u;
      if (!mbar_wait(&empty[st], ph ^ 1u)) {
        atomicOr(g.err, 1);
        break;
      }
      mbar_expect_tx(&full[st], kStageBytes);
      const uint32_t sa = sbase + st * kStageBytes;
      tma_load3(sa, &tmA, &full[st], c * BK, m0, g.a_shared ? 0 : z);
      tma_load3(sa + kTileBytes, &tmB, &full[st], c * BK, n0, z);
      last_par[st] = (int)ph;
    }
    for (int st = 0; st < kStages; ++st)  // copies in flight land before the CTA leaves
      if (last_par[st] >= 0 && !mbar_wait(&full[st], (uint32_t)last_par[st])) atomicOr(g.err, 8);
  } else if (work && warp == 1 && lane == 0) {
    // ---- MMA issuer
    for (int c = c0; c < c1; ++c) {
      const int i = c - c0, st = i % kStages;
      const uint32_t ph = (uint32_t)(i / kStages) & 1u;
      if (!mbar_wait(&full[st], ph)) {
        atomicOr(g.err, 2);
        break;
      }
      tc_fence_after();
      const uint32_t sa = sbase + st * kStageBytes;
      const uint64_t da = sw128_desc(sa), db = sw128_desc(sa + kTileBytes);
#pragma unroll
      for (int kk = 0; kk < BK / 16; ++kk) {
        const uint64_t adv = (uint64_t)(kk * 32) >> 4;  // 16 BF16 = 32 bytes along K
        mma_bf16_128(tbase, da + adv, db + adv, (c > c0 || kk > 0) ? 1u : 0u);
      }
      mma_commit(&empty[st]);
    }
    mma_commit(done);  // arrives once every MMA above has completed
  }
  // ---- epilogue: warp w holds accumulator rows 32 (w % 4) .. + 31, columns
  // 64 (w / 4) .. + 63, in chunks staged where the operand tiles were: every
  // copy has landed and every MMA has read its tiles once `done` has come.  N and
  // every row length are multiples of 16 values.  4,096 rows x 256 x 4 members: a hidden
  // layer 20 us with four warps and a row per lane, 14 now; its derivative 17.5, 13.6.
  bool have = work && mbar_wait(done, 0);
  have = __all_sync(0xffffffffu, have);
  if (work && !have && lane == 0) atomicOr(g.err, 4);
  tc_fence_after();
  const int m_w = m0 + warp % 4 * 32;
  const uint32_t lane_addr = tbase + ((uint32_t)(warp % 4 * 32) << 16);
  float* sm = reinterpret_cast<float*>(smem) + warp * kChunk * kRowF;
  if (have && m_w < g.M) {
    const int rows = min(kChunk, g.M - m_w);
#pragma unroll 1
    for (int cc = warp / 4 * 2; cc < warp / 4 * 2 + 2; ++cc) {
      const int nb = n0 + cc * kChunk;
      if (nb >= g.N) break;
      const int cols = min(kChunk, g.N - nb);
      float x[kChunk];
      {
        uint32_t v[32];
        tmem_ld32(lane_addr + (uint32_t)(cc * kChunk), v);
#pragma unroll
        for (int j = 0; j < 32; ++j) x[j] = __uint_as_float(v[j]);
      }
      if ((EPI == EPI_HIDDEN || EPI == EPI_LINEAR) && g.bias) {
        const float* bias = g.bias + z * g.sBias + nb;
#pragma unroll
        for (int q = 0; q < 8; ++q) {
          if (4 * q >= cols) break;
          const float4 b = *(const float4*)(bias + 4 * q);
          x[4 * q] += b.x; x[4 * q + 1] += b.y; x[4 * q + 2] += b.z; x[4 * q + 3] += b.w;
        }
      }
      if (EPI == EPI_DSILU) {
        float zp[kChunk];
        load_rows_f32(sm, zp, g.zprev + z * g.sZ + (int64_t)m_w * g.ldz + nb, g.ldz, rows, cols, lane);
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          float zq[8], sg[8];
#pragma unroll
          for (int j = 0; j < 8; ++j) zq[j] = zp[8 * q + j];
          sigm8(zq, sg);
#pragma unroll
          for (int j = 0; j < 8; ++j) x[8 * q + j] = x[8 * q + j] * (sg[j] * (1.0f + zq[j] * (1.0f - sg[j])));
        }
      }
      if (EPI != EPI_DSILU && g.outf) {
        float* o = g.outf + z * g.sOutf + (int64_t)m_w * g.ldf + nb;
        if (EPI == EPI_PARTIAL) o += split * g.sSplit;
        store_rows_f32(sm, x, o, g.ldf, rows, cols, lane);
      }
      if (EPI == EPI_HIDDEN) {
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          float xq[8], sg[8];
#pragma unroll
          for (int j = 0; j < 8; ++j) xq[j] = x[8 * q + j];
          sigm8(xq, sg);
#pragma unroll
          for (int j = 0; j < 8; ++j) x[8 * q + j] = xq[j] * sg[j];
        }
      }
      if (EPI == EPI_HIDDEN || EPI == EPI_DSILU)
        store_rows_bf16(sm, x, g.outh + z * g.sOuth + (int64_t)m_w * g.ldh + nb, g.ldh,
                        g.outhT ? g.outhT + z * g.sOuthT + (int64_t)nb * g.ldhT + m_w : nullptr, g.ldhT, rows, cols,
                        lane);
    }
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  if (warp == 0) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tbase), "r"(kTmemCols));
}

template <int EPI>
__global__ void __launch_bounds__(kThreads, 2)
    mlp_tc_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB, TcGemm g) {
  gemm_tile<EPI>(tmA, tmB, g, blockIdx.y, blockIdx.x, blockIdx.z);
}

// The weight gradients of every layer in one launch: alone, none of them fills the
// GPU (4,096 rows, 4 members: four launches 35 us, 21.5 in one).
struct WgradSet {
  CUtensorMap a[kWgradGemms], b[kWgradGemms];
  TcGemm g[kWgradGemms];
  int first[kWgradGemms + 1];  // first block of each, counting n tiles, then m tiles and splits
};
__global__ void __launch_bounds__(kThreads, 2) mlp_wgrad_kernel(const __grid_constant__ WgradSet w) {
  int l = 0;
  while (l + 1 < kWgradGemms && (int)blockIdx.x >= w.first[l + 1]) ++l;
  const int i = blockIdx.x - w.first[l], n_nt = (w.g[l].N + BN - 1) / BN;
  gemm_tile<EPI_PARTIAL>(w.a[l], w.b[l], w.g[l], i / n_nt, i % n_nt, blockIdx.y);
}

template <int EPI>
cudaError_t launch_epi(const CUtensorMap& ma, const CUtensorMap& mb, const TcGemm& g, int members, cudaStream_t s) {
  static std::atomic<uint64_t> attr{0};  // devices where the limit is set, shared by all contexts
  cudaError_t e = set_smem_once(attr, mlp_tc_kernel<EPI>, kSmem);
  if (e != cudaSuccess) return e;
  const int n_mt = (g.M + BM - 1) / BM;
  dim3 grid((unsigned)((g.N + BN - 1) / BN), (unsigned)(n_mt * g.k_split), (unsigned)members);
  mlp_tc_kernel<EPI><<<grid, kThreads, kSmem, s>>>(ma, mb, g);
  return cudaGetLastError();
}

}  // namespace

static cudaError_t gemm_maps(const TcOperand& A, const TcOperand& B, const TcGemm& g, int members, CUtensorMap* ma,
                             CUtensorMap* mb) {
  if ((A.ld * 2) % 16 || (B.ld * 2) % 16 || (A.member_stride * 2) % 16 || (B.member_stride * 2) % 16)
    return cudaErrorInvalidValue;
  // the epilogue's 16-byte accesses
  if (g.N % 8 || g.ldf % 4 || g.ldh % 8 || g.ldz % 4 || g.sOutf % 4 || g.sSplit % 4 || g.sOuth % 8 || g.sZ % 4 ||
      g.sBias % 4 || ((uintptr_t)g.outf | (uintptr_t)g.outh | (uintptr_t)g.zprev | (uintptr_t)g.bias) % 16)
    return cudaErrorInvalidValue;
  if (!make_map3(ma, A.ptr, g.K, A.ld, A.rows, g.a_shared ? 1 : members, A.member_stride) ||
      !make_map3(mb, B.ptr, g.K, B.ld, B.rows, members, B.member_stride))
    return cudaErrorInvalidValue;
  return cudaSuccess;
}

cudaError_t mlp_tc_wgrads(const TcOperand* A, const TcOperand* B, const TcGemm* g, int members, cudaStream_t s) {
  WgradSet w;
  w.first[0] = 0;
  for (int l = 0; l < kWgradGemms; ++l) {
    cudaError_t e = gemm_maps(A[l], B[l], g[l], members, &w.a[l], &w.b[l]);
    if (e != cudaSuccess) return e;
    w.g[l] = g[l];
    w.first[l + 1] = w.first[l] + (g[l].N + BN - 1) / BN * ((g[l].M + BM - 1) / BM) * g[l].k_split;
  }
  static std::atomic<uint64_t> attr{0};
  cudaError_t e = set_smem_once(attr, mlp_wgrad_kernel, kSmem);
  if (e != cudaSuccess) return e;
  mlp_wgrad_kernel<<<dim3((unsigned)w.first[kWgradGemms], (unsigned)members), kThreads, kSmem, s>>>(w);
  return cudaGetLastError();
}

cudaError_t mlp_tc_gemm(int epi, const TcOperand& A, const TcOperand& B, const TcGemm& g, int members,
                        cudaStream_t s) {
  if (g.M <= 0 || g.N <= 0 || g.K <= 0) return cudaSuccess;
  CUtensorMap ma, mb;
  cudaError_t e = gemm_maps(A, B, g, members, &ma, &mb);
  if (e != cudaSuccess) return e;
  switch (epi) {
    case EPI_HIDDEN: return launch_epi<EPI_HIDDEN>(ma, mb, g, members, s);
    case EPI_LINEAR: return launch_epi<EPI_LINEAR>(ma, mb, g, members, s);
    default: return launch_epi<EPI_DSILU>(ma, mb, g, members, s);
  }
}

}  // namespace abc
