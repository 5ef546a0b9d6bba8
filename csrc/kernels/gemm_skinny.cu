// bf16 GEMM for few rows: D[M, N] = A[M, K] * op(B) with M <= 128 (a linear layer at decode-sized token counts, or its input
// gradient).  The weights are what is read, once, so the kernel is laid out as a stream over them:
//
//   * operands exchanged: 128 output features (rows of the weight matrix) are the M side of tcgen05.mma and the input rows,
//     rounded up to 16, the N side, so no tensor work or shared memory is spent on padding rows to 128 or 256;
//   * K is split over the CTAs of a cluster (up to 8): the 64 feature tiles of an 8192-wide layer alone would leave more
//     than half of the 148 SMs without a load to issue.  Each CTA accumulates its share of K in TMEM, leaves the fp32 partial
//     tile in its own shared memory, and every CTA of the cluster adds up a share of the rows over distributed shared memory
//     in rank order: no workspace, no atomics, the same result every time;
//   * two CTAs per SM (about 100 KiB of operand ring each), so that a CTA's start and reduction pass behind its neighbour's
//     stream.
//
// Device time on one B200, cold L2 (us; single-CTA 128 x 256 tiles -> this kernel): 24 rows 8192 x 8192 71.7 -> 38.8,
// 128 rows 73.7 -> 43.0, 24 rows 512 -> 8192 inner 59.4 -> 14.3, 24 rows 2048 x 2048 26.7 -> 12.3, 24 rows of 50257 x 2048
// 61.4 -> 53.3.  With the weights' bytes at the copy rate those take 20, 20, 1.3, 1.3 and 31; an empty launch measures about
// 8 in the same loop.  From 129 rows on the CTA-pair kernel is as good or better (256 rows of 50257 x 2048: 61.5 against 96 with
// a form of this kernel for 256 rows).
#include <cuda.h>

#include <string>

#include "gemm_api.h"
#include "gemm_epilogue.cuh"
#include "launch.h"
#include "tc05.cuh"
#include "tensormap.h"

namespace pccl {

namespace {

namespace sk {
constexpr int TILE_F = 128, BK = 64, UMMA_K = 16;
constexpr int W_BYTES = TILE_F * BK * 2;              // 16 KiB
constexpr int MAX_STAGES = 8;
constexpr int NUM_THREADS = 256;                      // producer warp, MMA warp; all eight read TMEM and reduce
constexpr int RING_BYTES = 100 * 1024;
constexpr int SMEM_BYTES = RING_BYTES + 1024 + 256;

struct Barriers {
  uint64_t full[MAX_STAGES];
  uint64_t empty[MAX_STAGES];
  uint64_t done;
  uint32_t tmem_base;
  uint32_t abort;
};
}  // namespace sk

struct SkinnyArgs {
  void* D;
  void* D2;
  const __nv_bfloat16* bias;
  long long ldd;
  int M, N, num_kb, nb, stages;     // nb: input rows rounded up to 16
  uint32_t flags;
  uint32_t* status;
};

__device__ __forceinline__ float4 ld_cluster_f4(uint32_t cluster_addr) {
  float4 v;
  asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(cluster_addr) : "memory");
  return v;
}

// Four consecutive features of one output row: bias, residual, GELU, accumulation, store.
__device__ __forceinline__ void skinny_store(const SkinnyArgs& A, int row, int col, float4 s) {
  float v[4] = {s.x, s.y, s.z, s.w};
  const long long at = static_cast<long long>(row) * A.ldd + col;
  const bool full = col + 4 <= A.N;
  if (A.flags & GEMM_BIAS) {
#pragma unroll
    for (int i = 0; i < 4; ++i)
      if (full || col + i < A.N) v[i] += __bfloat162float(A.bias[col + i]);
  }
  if (A.flags & GEMM_OUT_F32) {
    if (A.flags & GEMM_GELU_INPLACE) {
#pragma unroll
      for (int i = 0; i < 4; ++i) v[i] = gemm::gelu_tanh(v[i]);
    }
    float* d = static_cast<float*>(A.D) + at;
    if (full) {
      if (A.flags & GEMM_ACCUMULATE) {
        const float4 o = *reinterpret_cast<const float4*>(d);
        v[0] += o.x; v[1] += o.y; v[2] += o.z; v[3] += o.w;
      }
      *reinterpret_cast<float4*>(d) = make_float4(v[0], v[1], v[2], v[3]);
    } else {
#pragma unroll
      for (int i = 0; i < 4; ++i)
        if (col + i < A.N) d[i] = (A.flags & GEMM_ACCUMULATE) ? d[i] + v[i] : v[i];
    }
    return;
  }
  __nv_bfloat16* d = static_cast<__nv_bfloat16*>(A.D) + at;
  __nv_bfloat16* d2 = static_cast<__nv_bfloat16*>(A.D2) + at;
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    if (!full && col + i >= A.N) continue;
    if (A.flags & GEMM_ADD_D2) v[i] += __bfloat162float(d2[i]);
    if (A.flags & GEMM_GELU_INPLACE) v[i] = gemm::gelu_tanh(v[i]);
    if (A.flags & GEMM_ACCUMULATE) v[i] += __bfloat162float(d[i]);
  }
  auto put = [&](__nv_bfloat16* o) {
    if (full) {
      const __nv_bfloat162 lo = __floats2bfloat162_rn(v[0], v[1]), hi = __floats2bfloat162_rn(v[2], v[3]);
      *reinterpret_cast<uint2*>(o) = make_uint2(*reinterpret_cast<const uint32_t*>(&lo), *reinterpret_cast<const uint32_t*>(&hi));
    } else {
#pragma unroll
      for (int i = 0; i < 4; ++i)
        if (col + i < A.N) o[i] = __float2bfloat16_rn(v[i]);
    }
  };
  put(d);
  if (A.flags & GEMM_GELU) {
#pragma unroll
    for (int i = 0; i < 4; ++i) v[i] = gemm::gelu_tanh(v[i]);
    put(d2);
  }
}

// Cluster of SPLITS CTAs along x: CTA rank r takes k-blocks [num_kb * r / SPLITS, num_kb * (r + 1) / SPLITS) of feature
// tile blockIdx.x / SPLITS.  W_MN: the weights are stored [K, N].
template <bool W_MN, int SPLITS>
__global__ void __launch_bounds__(sk::NUM_THREADS, 2)
gemm_skinny_kernel(const __grid_constant__ CUtensorMap tmW, const __grid_constant__ CUtensorMap tmX, const __grid_constant__ SkinnyArgs A) {
  using namespace sk;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~static_cast<uintptr_t>(1023));
  Barriers* bar = reinterpret_cast<Barriers*>(smem + RING_BYTES);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int rank = static_cast<int>(tc::cluster_ctarank());
  const int f0 = static_cast<int>(blockIdx.x) / SPLITS * TILE_F;
  const int kb0 = static_cast<int>(static_cast<long long>(A.num_kb) * rank / SPLITS);
  const int kb1 = static_cast<int>(static_cast<long long>(A.num_kb) * (rank + 1) / SPLITS);
  const int stage_bytes = W_BYTES + A.nb * (BK * 2);
  const uint32_t tmem_cols = A.nb <= 32 ? 32u : A.nb <= 64 ? 64u : 128u;
  volatile uint32_t* abort = &bar->abort;

  if (threadIdx.x == 0) {
    for (int s = 0; s < A.stages; ++s) {
      tc::mbar_init(&bar->full[s], 1);
      tc::mbar_init(&bar->empty[s], 1);
    }
    tc::mbar_init(&bar->done, 1);
    bar->abort = 0;
    tc::fence_barrier_init();
    tc::tma_prefetch_desc(&tmW);
    tc::tma_prefetch_desc(&tmX);
  }
  if (warp == 1) {
    tc::tmem_alloc(&bar->tmem_base, tmem_cols);
    tc::tmem_relinquish();
  }
  tc::tc_fence_before();
  __syncthreads();
  tc::tc_fence_after();
  const uint32_t tmem = bar->tmem_base;
  dev::pdl_launch();
  dev::pdl_wait();

  if (warp == 0) {
    if (tc::elect_one()) {
      int stage = 0;
      uint32_t phase = 0, armed = 0, armed_par = 0;
      bool ok = true;
      for (int kb = kb0; kb < kb1; ++kb) {
        if (!tc::mbar_wait(&bar->empty[stage], phase ^ 1, abort)) { ok = false; break; }
        uint8_t* sw = smem + stage * stage_bytes;
        tc::mbar_arrive_expect_tx(&bar->full[stage], static_cast<uint32_t>(stage_bytes));
        armed |= 1u << stage;
        armed_par = (armed_par & ~(1u << stage)) | (phase << stage);
        if constexpr (!W_MN) {
          tc::tma_load_2d(sw, &tmW, &bar->full[stage], kb * BK, f0);
        } else {
          tc::tma_load_2d(sw, &tmW, &bar->full[stage], f0, kb * BK);
          tc::tma_load_2d(sw + W_BYTES / 2, &tmW, &bar->full[stage], f0 + 64, kb * BK);
        }
        tc::tma_load_2d(sw + W_BYTES, &tmX, &bar->full[stage], kb * BK, 0);
        if (++stage == A.stages) { stage = 0; phase ^= 1; }
      }
      if (!ok) {
        if (atomicExch(const_cast<uint32_t*>(&bar->abort), 1u) == 0) dev::report(A.status, ST_TIMEOUT, blockIdx.x, 0, 0);
        for (int s = 0; s < A.stages; ++s)
          if (armed & (1u << s))
            for (uint32_t i = 0; i < (1u << 16) && !tc::mbar_try_wait(&bar->full[s], (armed_par >> s) & 1); ++i) {}
      }
    }
  } else if (warp == 1) {
    if (tc::elect_one()) {
      const uint32_t idesc = tc::make_idesc(1, 1, W_MN, false, TILE_F, static_cast<uint32_t>(A.nb));
      constexpr uint32_t W_LBO = W_MN ? 64 * BK * 2 : 16, W_KSTEP = W_MN ? (UMMA_K / 8) * 1024 : UMMA_K * 2;
      int stage = 0;
      uint32_t phase = 0;
      bool ok = true;
      for (int kb = kb0; kb < kb1; ++kb) {
        if (!tc::mbar_wait(&bar->full[stage], phase, abort)) { ok = false; break; }
        tc::tc_fence_after();
        const uint32_t sw = tc::smem_u32(smem + stage * stage_bytes), sx = sw + W_BYTES;
#pragma unroll
        for (int k = 0; k < BK / UMMA_K; ++k)
          tc::mma_f16(tmem, tc::smem_desc_sw128(sw + k * W_KSTEP, W_LBO, 1024), tc::smem_desc_sw128(sx + k * UMMA_K * 2, 16, 1024), idesc,
                      kb > kb0 || k > 0);
        tc::mma_commit(&bar->empty[stage]);
        if (++stage == A.stages) { stage = 0; phase ^= 1; }
      }
      if (!ok && atomicExch(const_cast<uint32_t*>(&bar->abort), 1u) == 0) dev::report(A.status, ST_TIMEOUT, blockIdx.x, 1, 0);
      tc::mma_commit(&bar->done);                   // every MMA above has retired: the ring is drained, the sums are complete
    }
  }
  __syncwarp();
  // every thread waits for the accumulator, then the ring becomes the partial tile
  if (!tc::mbar_wait(&bar->done, 0, abort) && lane == 0 && atomicExch(const_cast<uint32_t*>(&bar->abort), 1u) == 0)
    dev::report(A.status, ST_TIMEOUT, blockIdx.x, 2, 0);
  tc::tc_fence_after();
  __syncthreads();
  const bool failed = *abort != 0;

  float* P = reinterpret_cast<float*>(smem);        // [row][128 features], up to 64 KiB over the drained ring
  const uint32_t p_addr = tc::smem_u32(P);
  if (!failed) {                                    // two warps per lane quarter, each half of the rows
    const int quarter = warp & 3, half = (A.nb / 16 + 1) / 2 * 16;
    for (int c = (warp >> 2) ? half : 0; c < ((warp >> 2) ? A.nb : half); c += 16) {
      uint32_t r[16];
      tc::tmem_ld_32x16(tmem + (static_cast<uint32_t>(quarter * 32) << 16) + c, r);
      tc::tmem_ld_wait();
#pragma unroll
      for (int j = 0; j < 16; ++j) P[(c + j) * TILE_F + quarter * 32 + lane] = __uint_as_float(r[j]);
    }
  }
  tc::cluster_sync();                               // all partial tiles of the cluster are written
  if (!failed) {
    // a warp takes one row at a time per CTA of the cluster; eight 16-byte loads are in flight per lane
    constexpr int R = 8 / SPLITS;
    for (int row = rank + warp * SPLITS; row < A.M; row += 8 * SPLITS * R) {
      float4 v[R][SPLITS];
#pragma unroll
      for (int i = 0; i < R; ++i) {
        const int rr = min(row + i * 8 * SPLITS, A.M - 1);
        const uint32_t off = p_addr + static_cast<uint32_t>(rr * TILE_F + lane * 4) * 4u;
#pragma unroll
        for (int q = 0; q < SPLITS; ++q) v[i][q] = ld_cluster_f4(tc::mapa(off, static_cast<uint32_t>(q)));
      }
#pragma unroll
      for (int i = 0; i < R; ++i) {
        float4 s = v[i][0];
#pragma unroll
        for (int q = 1; q < SPLITS; ++q) {
          s.x += v[i][q].x; s.y += v[i][q].y; s.z += v[i][q].z; s.w += v[i][q].w;
        }
        if (row + i * 8 * SPLITS < A.M && f0 + lane * 4 < A.N) skinny_store(A, row + i * 8 * SPLITS, f0 + lane * 4, s);
      }
    }
  }
  tc::cluster_sync();                               // nobody reads this CTA's partials any more
  tc::tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    tc::tc_fence_after();
    tc::tmem_dealloc(tmem, tmem_cols);
  }
}

}  // namespace

// CTAs per feature tile: as many as are resident at once (two per SM), each with at least four k-blocks to stream.  Measured at 24
// rows with 1 / 2 / 4 / 8 CTAs per tile (us): 8192 x 8192 51 / 41 / 39 / 43, 12288 x 4096 35 / 31 / 37 / 39, 50257 x 2048
// 53 / 59 / 66 / 84, 512 x 8192 37 / 25 / 16 / 14: the rule takes 4, 2, 1 and 8.
int gemmSkinnySplits(int N, int K, int sms) {
  const int tiles = (N + sk::TILE_F - 1) / sk::TILE_F, num_kb = (K + sk::BK - 1) / sk::BK;
  int splits = 1;
  while (splits < 8 && tiles * splits * 2 <= 2 * sms && num_kb >= splits * 8) splits *= 2;
  return splits;
}

int gemmSkinnyBf16(const void* A, int64_t lda, const void* B, int64_t ldb, void* D, int64_t ldd, int M, int N, int K, uint32_t flags,
                   const void* bias, void* D2, uint32_t* status, cudaStream_t stream, std::string* err) {
  const bool w_mn = flags & GEMM_B_MN;
  const int nb = (M + 15) / 16 * 16;
  CUtensorMap tw, tx;
  if (!makeTensorMap2D(&tx, A, TM_BF16, K, M, lda, sk::BK, nb, err)) return static_cast<int>(cudaErrorInvalidValue);
  if (!w_mn ? !makeTensorMap2D(&tw, B, TM_BF16, K, N, ldb, sk::BK, sk::TILE_F, err) : !makeTensorMap2D(&tw, B, TM_BF16, N, K, ldb, 64, sk::BK, err))
    return static_cast<int>(cudaErrorInvalidValue);
  const int num_kb = (K + sk::BK - 1) / sk::BK;
  const int tiles = (N + sk::TILE_F - 1) / sk::TILE_F;
  int stages = sk::RING_BYTES / (sk::W_BYTES + nb * sk::BK * 2);
  if (stages > sk::MAX_STAGES) stages = sk::MAX_STAGES;
  const int splits = gemmSkinnySplits(N, K, deviceSmCount());
  SkinnyArgs args{D, D2, static_cast<const __nv_bfloat16*>(bias), ldd, M, N, num_kb, nb, stages, flags, status};
  static bool set[8] = {false, false, false, false, false, false, false, false};
  auto go = [&](auto kern, bool* done) {
    if (!*done) {
      cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, sk::SMEM_BYTES);
      if (e != cudaSuccess) return static_cast<int>(e);
      *done = true;
    }
    return static_cast<int>(launchOverlapped(kern, dim3(tiles * splits), dim3(sk::NUM_THREADS), sk::SMEM_BYTES, stream, splits, tw, tx, args));
  };
  switch (splits) {
    case 1: return w_mn ? go(gemm_skinny_kernel<true, 1>, set + 4) : go(gemm_skinny_kernel<false, 1>, set);
    case 2: return w_mn ? go(gemm_skinny_kernel<true, 2>, set + 5) : go(gemm_skinny_kernel<false, 2>, set + 1);
    case 4: return w_mn ? go(gemm_skinny_kernel<true, 4>, set + 6) : go(gemm_skinny_kernel<false, 4>, set + 2);
    default: return w_mn ? go(gemm_skinny_kernel<true, 8>, set + 7) : go(gemm_skinny_kernel<false, 8>, set + 3);
  }
}

}  // namespace pccl
