// Plain bf16 GEMM on the tcgen05 pipeline (see gemm_pipeline.cuh) with a fused epilogue:
// optional bias, optional GELU side output, bf16 or fp32 store, optional accumulation into D.
// The reference has no GEMM of any kind (cutlass and composable_kernel are empty submodules,
// .gitmodules:4-9); this is the "computation" half of its "communication & computation" claim.
#include <cuda.h>

#include <cstdlib>
#include <map>
#include <mutex>
#include <string>
#include <utility>

#include "gemm_api.h"
#include "gemm_epilogue.cuh"
#include "gemm_pipeline.cuh"
#include "gemm_pipeline2.cuh"
#include "launch.h"
#include "tensormap.h"

namespace pccl {

namespace {

using namespace gemm;

template <bool A_MN, bool B_MN>
__global__ void __launch_bounds__(NUM_THREADS, 1)
gemm_bf16_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB, StoreEpi epi, int K,
                 uint32_t* status) {
  GroupedSched sched{(epi.M + BM - 1) / BM, (epi.N + BN - 1) / BN, static_cast<int>(blockIdx.x), static_cast<int>(gridDim.x)};
  NoGate gate;
  run<A_MN, B_MN>(&tmA, &tmB, K, sched, gate, epi, status);
}

// ---- CTA-pair kernel ---------------------------------------------------------------------------------
// GroupedSched's order, handed out tile by tile at run time (gemm2::run, DYN): `counter` is a zeroed word that belongs to
// the launching stream.
struct DynGroupedSched {
  int tiles_m, tiles_n;
  uint32_t* counter;
  uint32_t total;
  __device__ __forceinline__ bool at(int idx, TileCoord* t) const {
    const int per_group = GroupedSched::GROUP_M * tiles_n;
    const int g = idx / per_group, r = idx % per_group;
    const int gm = min(GroupedSched::GROUP_M, tiles_m - g * GroupedSched::GROUP_M);
    t->m = g * GroupedSched::GROUP_M + r % gm;
    t->n = r / gm;
    t->extra = 0;
    return true;
  }
};

template <bool A_MN, bool B_MN, class Epi = StoreEpi, bool DYN = false>
__global__ void __launch_bounds__(gemm2::NUM_THREADS_WIDE, 1)
gemm_bf16_pair_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB, Epi epi, int K,
                      uint32_t* status, uint32_t* counter) {
  const int tiles_m = (epi.M + gemm2::PAIR_M - 1) / gemm2::PAIR_M, tiles_n = (epi.N + epi.bn - 1) / epi.bn;
  NoGate gate;
  const int cta = static_cast<int>(tc::cluster_ctarank());
  gemm2::PairEpi<Epi> pe{epi, cta};
  gemm2::PairGate<NoGate> pg{gate, cta};
  if constexpr (DYN) {
    DynGroupedSched sched{tiles_m, tiles_n, counter, static_cast<uint32_t>(tiles_m * tiles_n)};
    gemm2::run<A_MN, B_MN, DynGroupedSched, gemm2::PairGate<NoGate>, gemm2::PairEpi<Epi>, gemm2::STAGES, 1, true, 8>(&tmA, &tmB, K, sched, pg, pe, status);
  } else {
    GroupedSched sched{tiles_m, tiles_n, static_cast<int>(blockIdx.x >> 1), static_cast<int>(gridDim.x >> 1)};
    gemm2::run<A_MN, B_MN, GroupedSched, gemm2::PairGate<NoGate>, gemm2::PairEpi<Epi>, gemm2::STAGES, 1, false, 8>(&tmA, &tmB, K, sched, pg, pe, status);
  }
}

// ---- two GEMMs with one K as one tile list ---------------------------------------------------------------------------
struct DualMaps { CUtensorMap a[2], b[2]; };

struct DualSched {
  int tiles_m[2], tiles_n[2], first, stride;
  uint32_t* counter;       // dynamic scheduling: see DynGroupedSched; null = round-robin
  uint32_t total;
  __device__ __forceinline__ bool get(int it, TileCoord* t) const { return at(first + static_cast<long long>(it) * stride, t); }
  __device__ __forceinline__ bool at(long long idx, TileCoord* t) const {
    const long long n0 = static_cast<long long>(tiles_m[0]) * tiles_n[0];
    const int q = idx >= n0 ? 1 : 0;
    if (q) idx -= n0;
    const int tm = q ? tiles_m[1] : tiles_m[0], tn = q ? tiles_n[1] : tiles_n[0];       // no variable index: the arrays would live in local memory
    if (idx >= static_cast<long long>(tm) * tn) return false;
    const int per_group = GroupedSched::GROUP_M * tn;
    const int g = static_cast<int>(idx / per_group), r = static_cast<int>(idx % per_group);
    const int gm = min(GroupedSched::GROUP_M, tm - g * GroupedSched::GROUP_M);
    t->m = g * GroupedSched::GROUP_M + r % gm;
    t->n = r / gm;
    t->extra = q;
    return true;
  }
};

struct DualEpi {
  static constexpr bool kRow128 = false;
  StoreEpi e[2];
  StoreEpi cur;          // the tile's problem, picked once per tile: indexed with a variable the two would live in local memory
  __device__ __forceinline__ int width() const { return e[0].bn; }        // one width for both problems
  __device__ __forceinline__ int a_row0(const TileCoord& t) const { return e[0].a_row0(t); }
  __device__ __forceinline__ int b_row0(const TileCoord& t) const { return e[0].b_row0(t); }
  __device__ __forceinline__ void attach_smem(uint8_t*) {}
  __device__ __forceinline__ void attach_patch(uint8_t* p) { e[0].attach_patch(p); e[1].attach_patch(p); }
  __device__ __forceinline__ void tile_begin(const TileCoord& t) {
    cur = e[0];
    if (t.extra) cur = e[1];
  }
  __device__ __forceinline__ void tile_done(const TileCoord&, const volatile uint32_t*) {}
  __device__ __forceinline__ void strip(const TileCoord& t, int row, int col, uint32_t* r) { cur.strip(t, row, col, r); }
};

template <bool A_MN, bool B_MN, bool DYN>
__global__ void __launch_bounds__(gemm2::NUM_THREADS_WIDE, 1)
gemm_bf16_pair_dual_kernel(const __grid_constant__ DualMaps maps, DualEpi epi, int K, uint32_t* status, uint32_t* counter) {
  DualSched sched{{(epi.e[0].M + gemm2::PAIR_M - 1) / gemm2::PAIR_M, (epi.e[1].M + gemm2::PAIR_M - 1) / gemm2::PAIR_M},
                  {(epi.e[0].N + epi.e[0].bn - 1) / epi.e[0].bn, (epi.e[1].N + epi.e[1].bn - 1) / epi.e[1].bn},
                  static_cast<int>(blockIdx.x >> 1), static_cast<int>(gridDim.x >> 1), counter, 0u};
  sched.total = static_cast<uint32_t>(sched.tiles_m[0] * sched.tiles_n[0] + sched.tiles_m[1] * sched.tiles_n[1]);
  NoGate gate;
  const int cta = static_cast<int>(tc::cluster_ctarank());
  gemm2::PairEpi<DualEpi> pe{epi, cta};
  gemm2::PairGate<NoGate> pg{gate, cta};
  gemm2::run<A_MN, B_MN, DualSched, gemm2::PairGate<NoGate>, gemm2::PairEpi<DualEpi>, gemm2::STAGES, 2, DYN, 8>(maps.a, maps.b, K, sched, pg, pe, status);
}

thread_local std::string g_err;

// The zeroed counter word that dynamic tile scheduling of launches on `stream` uses (kernels on one stream run one after
// the other, and each leaves the word zeroed).  One 128-byte line per stream out of a pool made on first use; a null
// pointer (pool used up, or PCCL_GEMM_DYNAMIC=0) selects the round-robin kernels.
int g_dynamic = -1;      // -1: PCCL_GEMM_DYNAMIC decides (default on); 0 / 1: set by gemmSetDynamic
std::mutex g_counter_mu;
std::map<int, std::pair<uint32_t*, int>> g_counter_pools;      // device -> (base, lines handed out)
constexpr int kCounterPool = 64, kCounterStride = 32;          // lines per device, words per line

uint32_t* tileCounterFor(cudaStream_t stream) {
  static const bool env_off = std::getenv("PCCL_GEMM_DYNAMIC") && std::getenv("PCCL_GEMM_DYNAMIC")[0] == '0';
  if (g_dynamic == 0 || (g_dynamic < 0 && env_off)) return nullptr;
  constexpr int kPool = kCounterPool, kStride = kCounterStride;
  static std::map<std::pair<int, cudaStream_t>, uint32_t*> by_stream;
  auto& pools = g_counter_pools;
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) return nullptr;
  std::lock_guard<std::mutex> g(g_counter_mu);
  auto it = by_stream.find({dev, stream});
  if (it != by_stream.end()) return it->second;
  auto& pool = pools[dev];
  if (!pool.first) {
    cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
    if (cudaStreamIsCapturing(stream, &cap) != cudaSuccess || cap != cudaStreamCaptureStatusNone) return nullptr;
    uint32_t* base = nullptr;
    if (cudaMalloc(&base, kPool * kStride * sizeof(uint32_t)) != cudaSuccess) return nullptr;
    if (cudaMemset(base, 0, kPool * kStride * sizeof(uint32_t)) != cudaSuccess) return nullptr;
    pool = {base, 0};
  }
  if (pool.second >= kPool) return nullptr;
  uint32_t* p = pool.first + static_cast<size_t>(pool.second++) * kStride;
  by_stream[{dev, stream}] = p;
  return p;
}

// One CTA pair per cluster, allowed to start before the previous kernel of the stream has ended (launch.h).
template <class... KArgs, class... Args>
int launchPairKernel(void (*kern)(KArgs...), int grid, cudaStream_t stream, bool* attr_set, Args... args) {
  if (!*attr_set) {
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, gemm2::SMEM_BYTES);
    if (e != cudaSuccess) return static_cast<int>(e);
    *attr_set = true;
  }
  return static_cast<int>(launchOverlapped(kern, dim3(grid), dim3(gemm2::NUM_THREADS_WIDE), gemm2::SMEM_BYTES, stream, 2, args...));
}

template <bool A_MN, bool B_MN, class Epi = StoreEpi>
int launchPair(const CUtensorMap& ta, const CUtensorMap& tb, const Epi& epi, int K, int grid, uint32_t* status, cudaStream_t stream) {
  static bool attr_set = false, attr_set_dyn = false;
  uint32_t* counter = tileCounterFor(stream);
  return counter ? launchPairKernel(gemm_bf16_pair_kernel<A_MN, B_MN, Epi, true>, grid, stream, &attr_set_dyn, ta, tb, epi, K, status, counter)
                 : launchPairKernel(gemm_bf16_pair_kernel<A_MN, B_MN, Epi, false>, grid, stream, &attr_set, ta, tb, epi, K, status, counter);
}

template <bool A_MN, bool B_MN>
int launch(const CUtensorMap& ta, const CUtensorMap& tb, const StoreEpi& epi, int K, int grid, uint32_t* status, cudaStream_t stream) {
  static bool attr_set = false;
  auto kern = gemm_bf16_kernel<A_MN, B_MN>;
  if (!attr_set) {
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM_BYTES);
    if (e != cudaSuccess) return static_cast<int>(e);
    attr_set = true;
  }
  kern<<<grid, NUM_THREADS, SMEM_BYTES, stream>>>(ta, tb, epi, K, status);
  return static_cast<int>(cudaGetLastError());
}

}  // namespace

const char* gemmLastError() { return g_err.c_str(); }

// Tile width of a CTA-pair launch: 256 columns unless a narrower tile fills the last round of pairs better.  A round of
// narrower tiles is not cheaper in proportion -- every k-block still loads the pair's 256 rows of A, and L2 -> SM is what
// bounds it -- so the candidates are weighed with the measured time of a full round relative to a round of 256-wide tiles
// (16384 x 8192 x 2048 and 16384 x 2048 x 2048, one B200: 12.4 us at 256, 11.3 / 10.0 / 9.1 / 7.9 / 7.0 / 6.7 / 6.0 us at
// 224 ... 32).  Measured both ways (us, 256 wide -> chosen): 1531 x 2048 x 8192 53 -> 47 (48 tiles on 74 pairs -> 66),
// 2331 x 768 x 3072 28.6 -> 22.6, 8192 x 3584 x 8192 328 -> 316 (448 tiles = 6.05 rounds -> 512 = 6.9); 1531 x 6144 x 2048
// (144 tiles, 1.95 rounds) stays at 256: 40 against 44 at 192.  Two problems (gemmBf16Dual) share one width.
// With an MN-major B a CTA loads whole 64-column boxes, and a round costs more at the widths that do not fill them (1, .935, .84,
// .805, .70, .705, .68, .61 for 256 ... 32).  The one table serves that form and the epilogues with arithmetic too, because few
// choices lie between the two: over 20 shapes x 3 operand forms (768 x 2304 x 2331 to 8192 x 2048 x 16384), cold L2, the rule's width
// was never more than 4 % behind 256 columns and mostly the best of the eight or within 1 us of it (us, 256 -> rule; MN-major B:
// 1531 x 2048 x 8192 58 -> 50, 2331 x 768 x 3072 26.7 -> 21.5, 8192 x 3584 x 8192 366 -> 345, 1999 x 1416 x 3000 30.8 -> 31.7; GELU
// backward: 1000 x 1024 x 256 21.5 -> 15.4, 1531 x 8192 x 2048 51 -> 51 (224: 49), 8192 x 3584 x 8192 329 -> 331).
int gemmPairTileN(int tiles_m0, int n0, int tiles_m1, int n1, int pairs) {
  static const struct { int bn; float round; } kWidths[] = {{256, 1.f}, {224, .91f}, {192, .80f}, {160, .725f},
                                                            {128, .62f}, {96, .56f}, {64, .53f}, {32, .48f}};
  if (pairs < 1) pairs = 1;
  int best = 256;
  float best_cost = 0.f;
  for (const auto& w : kWidths) {
    const long long tiles = static_cast<long long>(tiles_m0) * ((n0 + w.bn - 1) / w.bn) + static_cast<long long>(tiles_m1) * ((n1 + w.bn - 1) / w.bn);
    const float cost = static_cast<float>((tiles + pairs - 1) / pairs) * w.round;
    if (w.bn == 256 || cost < best_cost * 0.999f) { best = w.bn; best_cost = cost; }
  }
  return best;
}

void gemmSetDynamic(int mode) { g_dynamic = mode < 0 ? -1 : (mode ? 1 : 0); }

int gemmResetTileCounters() {
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) return 0;
  std::lock_guard<std::mutex> g(g_counter_mu);
  auto it = g_counter_pools.find(dev);
  if (it == g_counter_pools.end() || !it->second.first) return 0;
  if (cudaDeviceSynchronize() != cudaSuccess) return static_cast<int>(cudaGetLastError());
  return static_cast<int>(cudaMemset(it->second.first, 0, kCounterPool * kCounterStride * sizeof(uint32_t)));
}

int gemmBf16(const void* A, int64_t lda, const void* B, int64_t ldb, void* D, int64_t ldd, int M, int N, int K,
             uint32_t flags, const void* bias, void* D2, int sms, uint32_t* status, cudaStream_t stream) {
  if (M <= 0 || N <= 0 || K <= 0) return 0;
  if ((lda | ldb | ldd) % 8 || (reinterpret_cast<uintptr_t>(A) | reinterpret_cast<uintptr_t>(B) | reinterpret_cast<uintptr_t>(D)) % 16) {
    g_err = "gemmBf16: strides must be multiples of 8 elements and pointers 16-byte aligned";
    return static_cast<int>(cudaErrorInvalidValue);
  }
  if ((flags & GEMM_ADD_D2) && (!D2 || (flags & (GEMM_OUT_F32 | GEMM_GELU)))) {
    g_err = "gemmBf16: the residual input needs D2 and a bf16 D, and excludes the GELU side output";
    return static_cast<int>(cudaErrorInvalidValue);
  }
  if ((flags & GEMM_GELU) && (!D2 || (flags & GEMM_OUT_F32))) {
    g_err = "gemmBf16: the GELU side output needs D2 and a bf16 D";
    return static_cast<int>(cudaErrorInvalidValue);
  }
  const bool a_mn = flags & GEMM_A_MN, b_mn = flags & GEMM_B_MN;
  if ((flags & GEMM_SKINNY) && !a_mn && M <= 128 && reinterpret_cast<uintptr_t>(D2) % 8 == 0)
    return gemmSkinnyBf16(A, lda, B, ldb, D, ldd, M, N, K, flags, bias, D2, status, stream, &g_err);
  // tensor maps: a K-major operand has dims {K, rows}, an MN-major one {rows, K}
  StoreEpi epi{D, D2, static_cast<const __nv_bfloat16*>(bias), ldd, M, N, flags};
  if (flags & GEMM_PAIR) {
    int n_sm2 = deviceSmCount();
    if (sms > 0 && sms < n_sm2) n_sm2 = sms;
    const int bn = gemmPairTileN((M + 255) / 256, N, 0, 0, n_sm2 / 2);
    epi.bn = bn;
    // per-CTA boxes: 128 rows of A and half of the tile's columns of B
    CUtensorMap pa, pb;
    if (!a_mn ? !makeTensorMap2D(&pa, A, TM_BF16, K, M, lda, BK, 128, &g_err) : !makeTensorMap2D(&pa, A, TM_BF16, M, K, lda, 64, BK, &g_err))
      return static_cast<int>(cudaErrorInvalidValue);
    if (!b_mn ? !makeTensorMap2D(&pb, B, TM_BF16, K, N, ldb, BK, bn / 2, &g_err) : !makeTensorMap2D(&pb, B, TM_BF16, N, K, ldb, 64, BK, &g_err))
      return static_cast<int>(cudaErrorInvalidValue);
    int pair_tiles = ((M + 255) / 256) * ((N + bn - 1) / bn);
    int grid2 = 2 * (pair_tiles < n_sm2 / 2 ? pair_tiles : n_sm2 / 2);
    if (a_mn) return b_mn ? launchPair<true, true>(pa, pb, epi, K, grid2, status, stream) : launchPair<true, false>(pa, pb, epi, K, grid2, status, stream);
    return b_mn ? launchPair<false, true>(pa, pb, epi, K, grid2, status, stream) : launchPair<false, false>(pa, pb, epi, K, grid2, status, stream);
  }
  CUtensorMap ta, tb;
  if (!a_mn ? !makeTensorMap2D(&ta, A, TM_BF16, K, M, lda, BK, BM, &g_err) : !makeTensorMap2D(&ta, A, TM_BF16, M, K, lda, 64, BK, &g_err))
    return static_cast<int>(cudaErrorInvalidValue);
  if (!b_mn ? !makeTensorMap2D(&tb, B, TM_BF16, K, N, ldb, BK, BN, &g_err) : !makeTensorMap2D(&tb, B, TM_BF16, N, K, ldb, 64, BK, &g_err))
    return static_cast<int>(cudaErrorInvalidValue);
  int tiles = ((M + BM - 1) / BM) * ((N + BN - 1) / BN);
  int n_sm = deviceSmCount();
  if (sms > 0 && sms < n_sm) n_sm = sms;
  int grid = tiles < n_sm ? tiles : n_sm;
  if (a_mn) return b_mn ? launch<true, true>(ta, tb, epi, K, grid, status, stream) : launch<true, false>(ta, tb, epi, K, grid, status, stream);
  return b_mn ? launch<false, true>(ta, tb, epi, K, grid, status, stream) : launch<false, false>(ta, tb, epi, K, grid, status, stream);
}

int gemmBf16Dgelu(const void* A, int64_t lda, const void* B, int64_t ldb, void* D, int64_t ldd, const void* pre, const ColSum& colsum,
                  int M, int N, int K, uint32_t flags, int sms, uint32_t* status, cudaStream_t stream) {
  if (M <= 0 || N <= 0 || K <= 0) return 0;
  if ((lda | ldb | ldd) % 8 || N % 32 ||
      (reinterpret_cast<uintptr_t>(A) | reinterpret_cast<uintptr_t>(B) | reinterpret_cast<uintptr_t>(D) | reinterpret_cast<uintptr_t>(pre)) % 16) {
    g_err = "gemmBf16Dgelu: N must be a multiple of 32, strides multiples of 8 elements, pointers 16-byte aligned";
    return static_cast<int>(cudaErrorInvalidValue);
  }
  const bool a_mn = flags & GEMM_A_MN, b_mn = flags & GEMM_B_MN;
  if (a_mn) {
    g_err = "gemmBf16Dgelu: an MN-major A operand is not built";
    return static_cast<int>(cudaErrorInvalidValue);
  }
  int n_sm = deviceSmCount();
  if (sms > 0 && sms < n_sm) n_sm = sms;
  const int bn = gemmPairTileN((M + 255) / 256, N, 0, 0, n_sm / 2);
  CUtensorMap pa, pb;
  if (!makeTensorMap2D(&pa, A, TM_BF16, K, M, lda, BK, 128, &g_err)) return static_cast<int>(cudaErrorInvalidValue);
  if (!b_mn ? !makeTensorMap2D(&pb, B, TM_BF16, K, N, ldb, BK, bn / 2, &g_err) : !makeTensorMap2D(&pb, B, TM_BF16, N, K, ldb, 64, BK, &g_err))
    return static_cast<int>(cudaErrorInvalidValue);
  const int pair_tiles = ((M + 255) / 256) * ((N + bn - 1) / bn);
  const int grid = 2 * (pair_tiles < n_sm / 2 ? pair_tiles : n_sm / 2);
  auto go = [&](auto epi) {
    using Epi = decltype(epi);
    return b_mn ? launchPair<false, true, Epi>(pa, pb, epi, K, grid, status, stream) : launchPair<false, false, Epi>(pa, pb, epi, K, grid, status, stream);
  };
  auto d = static_cast<__nv_bfloat16*>(D);
  auto x = static_cast<const __nv_bfloat16*>(pre);
  // Whole 256 x 256 tiles: gelu' through the hardware tanh.  Any other size had an accurate gelu' of its own before this epilogue
  // took it, and keeps one: 1 - tanh^2 cancels on the negative side, where the hardware tanh's 2^-11 is a fifth of gelu'(-3).
  float* parts = colsum.out ? colsum.parts : nullptr;
  const int e = M % 256 == 0 && N % 256 == 0 ? go(DgeluEpiT<false>{d, x, parts, ldd, M, N, bn}) : go(DgeluEpiT<true>{d, x, parts, ldd, M, N, bn});
  return e != 0 ? e : launchColSumParts(colsum, M, N, stream);
}

int gemmBf16Dual(const GemmProblem& p0, const GemmProblem& p1, int K, uint32_t flags, int sms, uint32_t* status, cudaStream_t stream) {
  const GemmProblem* ps[2] = {&p0, &p1};
  const bool a_mn = flags & GEMM_A_MN, b_mn = flags & GEMM_B_MN;
  if (K <= 0) return 0;
  int n_sm = deviceSmCount();
  if (sms > 0 && sms < n_sm) n_sm = sms;
  const int bn = gemmPairTileN((p0.M + 255) / 256, p0.N, (p1.M + 255) / 256, p1.N, n_sm / 2);
  DualMaps maps;
  DualEpi epi;
  for (int q = 0; q < 2; ++q) {
    const GemmProblem& p = *ps[q];
    if (p.M <= 0 || p.N <= 0 || (p.lda | p.ldb | p.ldd) % 8 ||
        (reinterpret_cast<uintptr_t>(p.A) | reinterpret_cast<uintptr_t>(p.B) | reinterpret_cast<uintptr_t>(p.D)) % 16) {
      g_err = "gemmBf16Dual: sizes must be positive, strides multiples of 8 elements, pointers 16-byte aligned";
      return static_cast<int>(cudaErrorInvalidValue);
    }
    if (!a_mn ? !makeTensorMap2D(&maps.a[q], p.A, TM_BF16, K, p.M, p.lda, BK, 128, &g_err) : !makeTensorMap2D(&maps.a[q], p.A, TM_BF16, p.M, K, p.lda, 64, BK, &g_err))
      return static_cast<int>(cudaErrorInvalidValue);
    if (!b_mn ? !makeTensorMap2D(&maps.b[q], p.B, TM_BF16, K, p.N, p.ldb, BK, bn / 2, &g_err) : !makeTensorMap2D(&maps.b[q], p.B, TM_BF16, p.N, K, p.ldb, 64, BK, &g_err))
      return static_cast<int>(cudaErrorInvalidValue);
    epi.e[q] = StoreEpi{p.D, nullptr, nullptr, p.ldd, p.M, p.N, (flags & GEMM_OUT_F32) | (p.accumulate ? GEMM_ACCUMULATE : 0u), bn};
  }
  const long long tiles = static_cast<long long>((p0.M + 255) / 256) * ((p0.N + bn - 1) / bn) + static_cast<long long>((p1.M + 255) / 256) * ((p1.N + bn - 1) / bn);
  const int grid = 2 * static_cast<int>(tiles < n_sm / 2 ? tiles : n_sm / 2);
  static bool attr_set[8] = {false, false, false, false, false, false, false, false};   // per kernel: the instantiations share one function type
  uint32_t* counter = tileCounterFor(stream);
  bool& attr = attr_set[(counter ? 4 : 0) | (a_mn ? 2 : 0) | (b_mn ? 1 : 0)];
  auto go = [&](auto kern) { return launchPairKernel(kern, grid, stream, &attr, maps, epi, K, status, counter); };
  if (counter) {
    if (a_mn) return b_mn ? go(gemm_bf16_pair_dual_kernel<true, true, true>) : go(gemm_bf16_pair_dual_kernel<true, false, true>);
    return b_mn ? go(gemm_bf16_pair_dual_kernel<false, true, true>) : go(gemm_bf16_pair_dual_kernel<false, false, true>);
  }
  if (a_mn) return b_mn ? go(gemm_bf16_pair_dual_kernel<true, true, false>) : go(gemm_bf16_pair_dual_kernel<true, false, false>);
  return b_mn ? go(gemm_bf16_pair_dual_kernel<false, true, false>) : go(gemm_bf16_pair_dual_kernel<false, false, false>);
}

}  // namespace pccl
