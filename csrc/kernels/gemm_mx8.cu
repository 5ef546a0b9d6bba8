// fp8 GEMM with hardware block scaling (gemm_mx8_pipeline.cuh) and the quantisers that produce its operands:
// e4m3 values with power-of-two (UE8M0) scales, one per row and 128 values of K for activations, one per
// 128 x 128 block for weights.  The reference has no GEMM and no quantiser.
#include <cuda.h>
#include <cuda_fp8.h>

#include <string>

#include "gemm_api.h"
#include "gemm_epilogue.cuh"
#include "gemm_mx8_pair.cuh"
#include "gemm_mx8_pipeline.cuh"
#include "tensormap.h"

namespace pccl {

namespace {

__global__ void __launch_bounds__(gemmx::NUM_THREADS, 1)
gemm_mx8_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB, gemm::StoreEpi epi,
                gemmx::Scales sc, int K, uint32_t* status) {
  gemm::GroupedSched sched{(epi.M + gemmx::BM - 1) / gemmx::BM, (epi.N + epi.bn - 1) / epi.bn, static_cast<int>(blockIdx.x),
                           static_cast<int>(gridDim.x)};
  gemm::NoGate gate;
  gemmx::run(&tmA, &tmB, K, sc, sched, gate, epi, status, epi.bn);
}

__global__ void __launch_bounds__(gemmxp::NUM_THREADS, 1)
gemm_mx8_pair_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB, gemm::StoreEpi epi,
                     gemmx::Scales sc, int K, uint32_t* status) {
  gemm::GroupedSched sched{(epi.M + gemmxp::PAIR_M - 1) / gemmxp::PAIR_M, (epi.N + epi.bn - 1) / epi.bn, static_cast<int>(blockIdx.x >> 1),
                           static_cast<int>(gridDim.x >> 1)};
  gemm2::PairEpi<gemm::StoreEpi> pe{epi, static_cast<int>(tc::cluster_ctarank())};
  gemmxp::run(&tmA, &tmB, K, sc, sched, pe, status);
}

// Smallest power of two >= amax / 448 (so that the scaled block fits e4m3), as a float and as its UE8M0 byte.
__device__ __forceinline__ float pow2_scale(float amax, uint8_t* byte) {
  if (!(amax > 0.f)) { *byte = 127; return 1.0f; }
  const float v = amax * (1.0f / 448.0f);
  uint32_t bits = __float_as_uint(v);
  uint32_t e = (bits >> 23) & 0xff;
  if (bits & 0x7fffff) e += 1;                 // round the mantissa up
  e = e < 1 ? 1 : (e > 254 ? 254 : e);
  *byte = static_cast<uint8_t>(e);
  return __uint_as_float(e << 23);
}

__device__ __forceinline__ uint2 quant8_mx(const float* f, float inv) {
  uint32_t w[2];
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    uint32_t lo = __nv_cvt_float2_to_fp8x2(make_float2(f[4 * h] * inv, f[4 * h + 1] * inv), __NV_SATFINITE, __NV_E4M3);
    uint32_t hi = __nv_cvt_float2_to_fp8x2(make_float2(f[4 * h + 2] * inv, f[4 * h + 3] * inv), __NV_SATFINITE, __NV_E4M3);
    w[h] = (lo & 0xffffu) | (hi << 16);
  }
  return make_uint2(w[0], w[1]);
}

// 16 consecutive lanes own one 1 x 128 block (8 values each); rows are whole blocks, so the matrix is one list of blocks.  PER
// loads in flight per thread (see quant_rows_kernel in moe.cu, its fp32-scale twin).  A CTA per row took 45 us at 8192 x 8192, this
// form 41: 201 MB at 4.9 TB/s.
template <int PER>
__global__ void __launch_bounds__(256) quant_rows_mx_kernel(const __nv_bfloat16* x, uint8_t* q,
                                                            uint8_t* scales, long long nvec) {
  dev::pdl_launch();
  dev::pdl_wait();
  constexpr int CHUNK = 256 * PER;
  for (long long v0 = static_cast<long long>(blockIdx.x) * CHUNK + threadIdx.x; v0 - (threadIdx.x & 31) < nvec; v0 += static_cast<long long>(gridDim.x) * CHUNK) {
    dev::Vec16 in[PER];
#pragma unroll
    for (int j = 0; j < PER; ++j)
      if (v0 + j * 256 < nvec) in[j] = dev::ld16(x + (v0 + j * 256) * 8);
#pragma unroll
    for (int j = 0; j < PER; ++j) {
      const long long v = v0 + j * 256;
      float f[8];
      float amax = 0.f;
      if (v < nvec) {
        dev::unpack<DT_BF16>(in[j], f);
#pragma unroll
        for (int i = 0; i < 8; ++i) amax = fmaxf(amax, fabsf(f[i]));
      }
#pragma unroll
      for (int o = 8; o > 0; o >>= 1) amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, o));
      uint8_t byte;
      const float scale = pow2_scale(amax, &byte);
      if (v < nvec) {
        *reinterpret_cast<uint2*>(q + v * 8) = quant8_mx(f, 1.0f / scale);
        if ((v & 15) == 0) scales[v >> 4] = byte;
      }
    }
  }
}

// one CTA per 128 x 128 block of a weight matrix
__global__ void __launch_bounds__(256) quant_blocks_mx_kernel(const __nv_bfloat16* __restrict__ w, uint8_t* __restrict__ q,
                                                              uint8_t* __restrict__ scales, int rows, int cols) {
  __shared__ float red[8];
  const int bc = blockIdx.x, br = blockIdx.y;
  const __nv_bfloat16* base = w + static_cast<long long>(br) * 128 * cols + bc * 128;
  float f[8][8];
  float amax = 0.f;
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    const int idx = threadIdx.x + i * 256, r = idx >> 4, v = idx & 15;
    dev::unpack<DT_BF16>(dev::ld16(base + static_cast<long long>(r) * cols + v * 8), f[i]);
#pragma unroll
    for (int j = 0; j < 8; ++j) amax = fmaxf(amax, fabsf(f[i][j]));
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, o));
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = amax;
  __syncthreads();
  amax = red[0];
#pragma unroll
  for (int i = 1; i < 8; ++i) amax = fmaxf(amax, red[i]);
  uint8_t byte;
  const float scale = pow2_scale(amax, &byte);
  if (threadIdx.x == 0) scales[br * (cols >> 7) + bc] = byte;
  const float inv = 1.0f / scale;
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    const int idx = threadIdx.x + i * 256, r = idx >> 4, v = idx & 15;
    *reinterpret_cast<uint2*>(q + (static_cast<long long>(br) * 128 + r) * cols + bc * 128 + v * 8) = quant8_mx(f[i], inv);
  }
}

thread_local std::string g_errx;

}  // namespace

const char* gemmMx8LastError() { return g_errx.c_str(); }

// Columns per tile: 224 unless narrower tiles fill the last round of CTAs better.  Measured time of a full round relative to
// 224 columns (148 tiles of 128 rows each, K = 2048 and 8192, one B200, mean of the two): a round is bound by the operands
// that an SM gets from L2, of which A's 128 rows stay.  1531 x 3584 x 8192: 192 tiles of 224 in two rounds, 276 of 160 in two.
// Against 224 columns (us): 300 x 4096 x 1024 15.3 -> 13.3, 777 x 2048 x 2048 19.5 -> 17.4, 1000 x 1152 x 4096 25.6 -> 21.4,
// 1531 x 3584 x 8192 60 -> 54 to 58; within 2 % at four larger shapes, which keep 224.
// Up to 32 rows all CTAs ask for the same few lines of A at the same time, and more of them queue longer: 1 x 8192 x 3584 takes 20.3
// with 224 columns, 20.5 with 160 and 24.4 with 64, 16 x 4096 x 7168 26.9, 24.6 and 28.7; from 40 rows on 64 columns are the best
// (40 x 8192 x 3584 20.2, 18.5, 18.1; 40 x 4096 x 7168 26.6, 24.6, 22.8).
struct RoundCost { int bn; float round; };
static int cheapestWidth(const RoundCost* widths, int count, int tiles_m, int n, int slots, int least, float* cost, long long* rounds) {
  int best = 0;
  for (int i = 0; i < count && widths[i].bn >= least; ++i) {
    const long long r = (static_cast<long long>(tiles_m) * ((n + widths[i].bn - 1) / widths[i].bn) + slots - 1) / slots;
    const float c = static_cast<float>(r) * widths[i].round;
    if (i == 0 || c < *cost * 0.999f) { best = widths[i].bn; *cost = c; *rounds = r; }
  }
  return best;
}
static int singleWidth(int rows, int n, int sms, float* cost, long long* rounds) {
  static const RoundCost kWidths[] = {{224, 1.f}, {192, .89f}, {160, .83f}, {128, .78f}, {96, .75f}, {64, .70f}, {32, .68f}};
  return cheapestWidth(kWidths, 7, (rows + gemmx::BM - 1) / gemmx::BM, n, sms, rows <= 32 ? 160 : 32, cost, rounds);
}
int gemmMx8TileN(int rows, int n, int sms) {
  float cost;
  long long rounds;
  return singleWidth(rows, n, sms, &cost, &rounds);
}

// Columns per tile of a CTA-pair launch, or 0 where single CTAs are the better form.  Pairs halve what an SM fetches of B: a full round
// of 74 pairs of 224 columns took 10.5 us at K = 3584 where 148 single CTAs took 13.0, 21.9 and 26 at K = 8192 (narrower tiles:
// mean of the two, relative).  A K block of theirs is a longer chain (barriers across the cluster), so what fits into one round of
// single CTAs stays there: 777 x 2048 x 2048 14.5 us single, 16.4 pairs; 384 x 8192 x 2048 16.4 and 18.5; 512 x 8192 x 8192 36.9 and 37.7.
// More than a round (us, cold L2, single -> pairs): 8192 x 3584 x 8192 180 -> 150, 8192 x 8192 x 3584 202 -> 159, 16384 x 8192 x 8192
// 851 -> 711 (3.06 PFLOP/s), 1531 x 8192 x 3584 46 -> 42, 1531 x 3584 x 8192 50 -> 46, 5000 x 1920 x 2048 31.4 -> 26.6, 640 x 7168 x 4096
// 30.6 -> 29.5, 1000 x 4096 x 4096 28.7 -> 26.7.
int gemmMx8PairTileN(int rows, int n, int sms) {
  static const RoundCost kWidths[] = {{224, 1.f}, {192, .90f}, {160, .84f}, {128, .76f}, {96, .69f}, {64, .66f}};
  float single, pair;
  long long single_rounds, pair_rounds;
  singleWidth(rows, n, sms, &single, &single_rounds);
  if (single_rounds < 2 || sms < 2) return 0;
  const int bn = cheapestWidth(kWidths, 6, (rows + gemmxp::PAIR_M - 1) / gemmxp::PAIR_M, n, sms / 2, 64, &pair, &pair_rounds);
  return pair < 1.2f * single ? bn : 0;
}

int launchQuantMx8Rows(const void* x, void* q, uint8_t* scales, long long rows, int k, cudaStream_t stream) {
  if (k % 128 || rows <= 0) return static_cast<int>(cudaErrorInvalidValue);
  const long long nvec = rows * (k >> 3), most = deviceSmCount() * 8ll;       // 256-thread CTAs resident at once
  auto go = [&](auto kern, long long blocks) {
    return static_cast<int>(launchOverlapped(kern, dim3(static_cast<unsigned>(blocks < most ? blocks : most)), dim3(256), 0, stream, 1,
                                             static_cast<const __nv_bfloat16*>(x), static_cast<uint8_t*>(q), scales, nvec));
  };
  return nvec <= most * 256 ? go(quant_rows_mx_kernel<1>, (nvec + 255) / 256) : go(quant_rows_mx_kernel<4>, (nvec + 1023) / 1024);
}

int launchQuantMx8Blocks(const void* w, void* q, uint8_t* scales, int rows, int cols, cudaStream_t stream) {
  if (rows % 128 || cols % 128 || rows <= 0 || cols <= 0) return static_cast<int>(cudaErrorInvalidValue);
  dim3 grid(cols / 128, rows / 128);
  quant_blocks_mx_kernel<<<grid, 256, 0, stream>>>(static_cast<const __nv_bfloat16*>(w), static_cast<uint8_t*>(q), scales, rows, cols);
  return static_cast<int>(cudaGetLastError());
}

int gemmMx8(const void* A, int64_t lda, const uint8_t* sa, int ld_sa, const void* B, int64_t ldb, const uint8_t* sb, int ld_sb,
            void* D, int64_t ldd, int M, int N, int K, uint32_t flags, const void* bias, void* D2, int sms, uint32_t* status,
            cudaStream_t stream) {
  if (M <= 0 || N <= 0 || K <= 0) return 0;
  if ((lda | ldb) % 16 || ldd % 8 || K % 128 ||
      (reinterpret_cast<uintptr_t>(A) | reinterpret_cast<uintptr_t>(B) | reinterpret_cast<uintptr_t>(D)) % 16) {
    g_errx = "gemmMx8: K must be a multiple of 128, operand strides multiples of 16, pointers 16-byte aligned";
    return static_cast<int>(cudaErrorInvalidValue);
  }
  if (flags & (GEMM_A_MN | GEMM_B_MN | GEMM_PAIR)) {
    g_errx = "gemmMx8: operands are K-major, and the launch itself picks single CTAs or pairs";
    return static_cast<int>(cudaErrorInvalidValue);
  }
  if ((flags & GEMM_GELU) && (!D2 || (flags & GEMM_OUT_F32))) {
    g_errx = "gemmMx8: the GELU side output needs D2 and a bf16 D";
    return static_cast<int>(cudaErrorInvalidValue);
  }
  if (ld_sa < K / 128 || ld_sb < K / 128) {
    g_errx = "gemmMx8: scale rows are shorter than K / 128";
    return static_cast<int>(cudaErrorInvalidValue);
  }
  CUtensorMap ta, tb;
  if (!makeTensorMap2D(&ta, A, TM_U8, K, M, lda, gemmx::BK, gemmx::BM, &g_errx)) return static_cast<int>(cudaErrorInvalidValue);
  int n_sm = deviceSmCount();
  if (sms > 0 && sms < n_sm) n_sm = sms;
  if (const int bn = gemmMx8PairTileN(M, N, n_sm)) {
    if (!makeTensorMap2D(&tb, B, TM_U8, K, N, ldb, gemmxp::BK, bn / 2, &g_errx)) return static_cast<int>(cudaErrorInvalidValue);
    static bool pair_attr_set = false;
    if (!pair_attr_set) {
      cudaError_t e = cudaFuncSetAttribute(gemm_mx8_pair_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, gemmxp::SMEM_BYTES);
      if (e != cudaSuccess) return static_cast<int>(e);
      pair_attr_set = true;
    }
    const int pair_tiles = ((M + gemmxp::PAIR_M - 1) / gemmxp::PAIR_M) * ((N + bn - 1) / bn), pairs = n_sm / 2;
    return static_cast<int>(launchOverlapped(gemm_mx8_pair_kernel, dim3(2 * (pair_tiles < pairs ? pair_tiles : pairs)), dim3(gemmxp::NUM_THREADS),
                                             gemmxp::SMEM_BYTES, stream, 2, ta, tb,
                                             gemm::StoreEpi{D, D2, static_cast<const __nv_bfloat16*>(bias), ldd, M, N, flags, bn},
                                             gemmx::Scales{sa, sb, ld_sa, ld_sb, M, N}, K, status));
  }
  const int bn = gemmMx8TileN(M, N, n_sm);
  if (!makeTensorMap2D(&tb, B, TM_U8, K, N, ldb, gemmx::BK, bn, &g_errx)) return static_cast<int>(cudaErrorInvalidValue);
  gemm::StoreEpi epi{D, D2, static_cast<const __nv_bfloat16*>(bias), ldd, M, N, flags, bn};
  gemmx::Scales sc{sa, sb, ld_sa, ld_sb, M, N};
  static bool attr_set = false;
  if (!attr_set) {
    cudaError_t e = cudaFuncSetAttribute(gemm_mx8_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, gemmx::SMEM_BYTES);
    if (e != cudaSuccess) return static_cast<int>(e);
    attr_set = true;
  }
  const int tiles = ((M + gemmx::BM - 1) / gemmx::BM) * ((N + bn - 1) / bn);
  return static_cast<int>(launchOverlapped(gemm_mx8_kernel, dim3(tiles < n_sm ? tiles : n_sm), dim3(gemmx::NUM_THREADS), gemmx::SMEM_BYTES, stream, 1,
                                           ta, tb, epi, sc, K, status));
}

}  // namespace pccl
