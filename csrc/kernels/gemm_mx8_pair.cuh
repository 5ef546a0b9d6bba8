// CTA-pair variant of the hardware-scaled fp8 pipeline (gemm_mx8_pipeline.cuh): two CTAs of a cluster (cta_group::2) compute one
// tile of 256 rows x up to 224 columns.  The single-CTA form is bound by the operands that an SM gets from L2: 44 KiB per K block of
// 128 x 224 outputs, 700 clocks at 63 bytes per clock where the tensor core needs 450.  Here a CTA fetches its own 128 rows of A and
// half of the tile's columns of B, 30 KiB per K block.
//
//   warp 0      TMA producer (both CTAs)
//   warp 1      MMA issuer (leader CTA): four MMAs 256 x width x 32 per stage; every fourth stage tcgen05.cp (cta_group::2) first brings
//               the scale images of the next 512 values of K from both CTAs' shared memory into both CTAs' TMEM
//   warp 2      scale builder (both CTAs): an image holds this CTA's 128 rows of A and ALL columns of the tile (the instruction wants
//               B's scales in full on either side)
//   warps 4..11 epilogue: two per TMEM lane quarter, each half of the tile's strips
//
// TMEM columns, bounded waits (and the wait for loads in flight when a role gives up) and the absence of multicast loads as in the single-CTA form.
#pragma once
#include "gemm_mx8_pipeline.cuh"
#include "gemm_pipeline2.cuh"

namespace pccl {
namespace gemmxp {

using gemm::TileCoord;
using gemmx::SF_BYTES;
using gemmx::SF_IMAGES;

constexpr int BM = 128, PAIR_M = 256, BN = gemmx::BN, BK = 128, UMMA_K = 32;
constexpr int STAGES = 6;
constexpr int A_BYTES = BM * BK, STAGE_BYTES = A_BYTES + BN / 2 * BK;      // 30 KiB
constexpr int TMEM_COLS = 512;
constexpr int EPI_WARPS = 8, FIRST_EPI_WARP = 4;
constexpr int NUM_THREADS = (FIRST_EPI_WARP + EPI_WARPS) * 32;
constexpr int BAR_BYTES = 256;
constexpr int SF_OFFSET = STAGES * STAGE_BYTES, BAR_OFFSET = SF_OFFSET + SF_IMAGES * SF_BYTES, PATCH_OFFSET = BAR_OFFSET + BAR_BYTES;
constexpr int SMEM_BYTES = PATCH_OFFSET + EPI_WARPS * gemm::kPatchBytes + 1024;
static_assert(SMEM_BYTES <= 232448, "shared memory budget");

struct Barriers {
  uint64_t full[STAGES];          // used in the leader: both CTAs' loads of the stage have landed
  uint64_t empty[STAGES];         // per CTA: the MMAs that read this stage have retired
  uint64_t tmem_full[2];          // per CTA: accumulator ready
  uint64_t tmem_empty[2];         // used in the leader: both CTAs' epilogues have drained the accumulator
  uint64_t sf_full[SF_IMAGES];    // used in the leader: both CTAs' scale images are written
  uint64_t sf_empty[SF_IMAGES];   // per CTA: the MMAs of that group of K blocks have retired
  uint64_t drain;
  uint32_t tmem_base;
  uint32_t abort;
};
static_assert(sizeof(Barriers) <= BAR_BYTES, "barriers overrun their area");

__device__ __forceinline__ void tmem_cp_32x128b_x4_pair(uint32_t taddr, uint64_t desc) {
  asm volatile("tcgen05.cp.cta_group::2.32x128b.warpx4 [%0], %1;" ::"r"(taddr), "l"(desc) : "memory");
}
__device__ __forceinline__ void mma_mx8_pair(uint32_t d_tmem, uint64_t a_desc, uint64_t b_desc, uint32_t idesc, uint32_t tsfa, uint32_t tsfb,
                                             uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::2.kind::mxf8f6f4.block_scale [%0], %1, %2, %3, [%5], [%6], p;\n\t}\n"
      ::"r"(d_tmem), "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(accumulate), "r"(tsfa), "r"(tsfb)
      : "memory");
}

// `sched` enumerates pair tiles (t.m: 256-row blocks, t.n: blocks of epi.width() columns); `epi` is a gemm2::PairEpi.
template <class Sched, class Epi>
__device__ __forceinline__ void run(const CUtensorMap* tmA, const CUtensorMap* tmB, int K, const gemmx::Scales& sc, const Sched& sched, Epi& epi,
                                    uint32_t* status) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~static_cast<uintptr_t>(1023));
  uint8_t* sf_smem = smem + SF_OFFSET;
  Barriers* bar = reinterpret_cast<Barriers*>(smem + BAR_OFFSET);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const bool leader = tc::cluster_ctarank() == 0;
  const int num_kb = (K + BK - 1) / BK, num_kg = (num_kb + 3) / 4;
  const int width = epi.width();
  volatile uint32_t* abort = &bar->abort;

  if (threadIdx.x == 0) {
    for (int s = 0; s < STAGES; ++s) {
      tc::mbar_init(&bar->full[s], 1);
      tc::mbar_init(&bar->empty[s], 1);
    }
    for (int a = 0; a < 2; ++a) {
      tc::mbar_init(&bar->tmem_full[a], 1);
      tc::mbar_init(&bar->tmem_empty[a], 2 * EPI_WARPS);
    }
    for (int a = 0; a < SF_IMAGES; ++a) {
      tc::mbar_init(&bar->sf_full[a], 2);
      tc::mbar_init(&bar->sf_empty[a], 1);
    }
    tc::mbar_init(&bar->drain, 1);
    bar->abort = 0;
    tc::fence_barrier_init();
    tc::tma_prefetch_desc(tmA);
    tc::tma_prefetch_desc(tmB);
  }
  __syncthreads();
  tc::cluster_sync();                 // the peer's barriers are initialised before anything signals them
  if (warp == 1) {
    tc::tmem_alloc_pair(&bar->tmem_base, TMEM_COLS);
    tc::tmem_relinquish_pair();
  }
  tc::tc_fence_before();
  __syncthreads();
  tc::tc_fence_after();
  const uint32_t tmem = bar->tmem_base;
  dev::pdl_wait();                    // nothing above touched global memory
  epi.attach_patch(smem + PATCH_OFFSET - (FIRST_EPI_WARP - 2) * gemm::kPatchBytes);      // my_patch() counts from warp 2

  if (warp == 0) {
    // ------------------------------------------------------------------ TMA producer (both CTAs)
    if (tc::elect_one()) {
      const uint32_t stage_tx = 2u * (A_BYTES + static_cast<uint32_t>(width / 2) * BK);      // both CTAs' bytes
      int stage = 0;
      uint32_t phase = 0;
      bool ok = true;
      TileCoord t;
      for (int it = 0; ok && sched.get(it, &t); ++it) {
        const int row0 = epi.a_row0(t), col0 = epi.b_row0(t);        // already offset by this CTA's half
        for (int kb = 0; kb < num_kb; ++kb) {
          if (!tc::mbar_wait(&bar->empty[stage], phase ^ 1, abort)) { ok = false; break; }
          uint8_t* sa = smem + stage * STAGE_BYTES;
          const uint32_t full_leader = tc::mapa(tc::smem_u32(&bar->full[stage]), 0);
          if (leader) tc::mbar_arrive_expect_tx(&bar->full[stage], stage_tx);
          tc::tma_load_2d_pair(sa, tmA, full_leader, kb * BK, row0);
          tc::tma_load_2d_pair(sa + A_BYTES, tmB, full_leader, kb * BK, col0);
          if (++stage == STAGES) { stage = 0; phase ^= 1; }
        }
      }
      if (!ok && atomicExch(const_cast<uint32_t*>(&bar->abort), 1u) == 0) dev::report(status, ST_TIMEOUT, blockIdx.x, 0, 0);
      dev::pdl_launch();                // the last load is on its way: the next kernel of the stream may move in
    }
  } else if (warp == 1) {
    // ------------------------------------------------------------------ MMA issuer (leader CTA only)
    if (leader && tc::elect_one()) {
      const uint32_t idesc0 = gemmx::make_idesc_mx(PAIR_M, static_cast<uint32_t>(width));
      int stage = 0, acc = 0;
      uint32_t phase = 0, acc_phase = 0, g = 0;       // g: 512-wide K groups issued so far
      bool ok = true;
      TileCoord t;
      for (int it = 0; ok && sched.get(it, &t); ++it) {
        if (!tc::mbar_wait(&bar->tmem_empty[acc], acc_phase ^ 1, abort)) { ok = false; break; }
        tc::tc_fence_after();
        const uint32_t d_tmem = tmem + acc * 256;
        for (int kb = 0; kb < num_kb; ++kb) {
          // group g: image and TMEM words g & 1; why a copy cannot overwrite words in use: see the single-CTA form
          const uint32_t im = g & 1, tsfa = tmem + BN + 16 * im, tsfb = tsfa + 4;
          if (!tc::mbar_wait(&bar->full[stage], phase, abort)) { ok = false; break; }
          if ((kb & 3) == 0) {
            if (!tc::mbar_wait(&bar->sf_full[im], (g >> 1) & 1, abort)) { ok = false; break; }      // the peer wrote its image
            tc::tc_fence_after();
            const uint32_t img = tc::smem_u32(sf_smem + im * SF_BYTES);
            tmem_cp_32x128b_x4_pair(tsfa, gemmx::sf_desc(img));
            tmem_cp_32x128b_x4_pair(tsfb, gemmx::sf_desc(img + 512));
            tmem_cp_32x128b_x4_pair(tsfb + 4, gemmx::sf_desc(img + 1024));
          }
          tc::tc_fence_after();
          const uint32_t sa = tc::smem_u32(smem + stage * STAGE_BYTES), sb = sa + A_BYTES;
          const uint32_t sf = static_cast<uint32_t>(kb & 3);
          const uint32_t idesc = idesc0 | (sf << 29) | (sf << 4);
#pragma unroll
          for (int k = 0; k < BK / UMMA_K; ++k)
            mma_mx8_pair(d_tmem, tc::smem_desc_sw128(sa + k * UMMA_K, 16, 1024), tc::smem_desc_sw128(sb + k * UMMA_K, 16, 1024), idesc, tsfa, tsfb,
                         (kb | k) != 0);
          tc::mma_commit_pair(&bar->empty[stage], 3);          // frees the stage in both CTAs
          if (++stage == STAGES) { stage = 0; phase ^= 1; }
          if ((kb & 3) == 3 || kb == num_kb - 1) {
            tc::mma_commit_pair(&bar->sf_empty[im], 3);
            ++g;
          }
        }
        if (!ok) break;
        tc::mma_commit_pair(&bar->tmem_full[acc], 3);          // accumulator ready in both CTAs
        if (++acc == 2) { acc = 0; acc_phase ^= 1; }
      }
      if (!ok) {
        if (atomicExch(const_cast<uint32_t*>(&bar->abort), 1u) == 0) dev::report(status, ST_TIMEOUT, blockIdx.x, 1, 0);
        tc::drain_pair_loads(bar->full, STAGES, stage, phase);
      }
      tc::mma_commit_pair(&bar->drain, 1);
      for (uint32_t i = 0; i < (1u << 20) && !tc::mbar_try_wait(&bar->drain, 0); ++i) {}
    }
  } else if (warp == 2) {
    // ------------------------------------------------------------------ scale builder (both CTAs)
    // The words of the NEXT group (also across a tile boundary) are in flight while the MMAs of the current ones run.
    gemmx::ScaleWords words;
    auto fetch = [&](const TileCoord& tt, int kg) { words.fetch(sc, epi.a_row0(tt), tt.n * width, kg * 4, num_kb, lane); };
    uint32_t g = 0;
    bool ok = true;
    TileCoord t, tn;
    bool have = sched.get(0, &t);
    if (have) fetch(t, 0);
    for (int it = 0; ok && have; ++it) {
      const bool have_next = sched.get(it + 1, &tn);
      for (int kg = 0; kg < num_kg; ++kg, ++g) {
        const uint32_t im = g & 1;
        int open = 1;
        if (lane == 0) open = tc::mbar_wait(&bar->sf_empty[im], ((g >> 1) & 1) ^ 1, abort) ? 1 : 0;
        if (!__shfl_sync(0xffffffffu, open, 0)) { ok = false; break; }
        words.store(sf_smem + im * SF_BYTES, lane);
        tc::fence_proxy_async_smem();                // the image is read by tcgen05.cp (async proxy)
        __syncwarp();
        if (lane == 0) tc::mbar_arrive_remote(tc::mapa(tc::smem_u32(&bar->sf_full[im]), 0));     // on the leader's barrier
        if (kg + 1 < num_kg) fetch(t, kg + 1);
        else if (have_next) fetch(tn, 0);
      }
      t = tn;
      have = have_next;
    }
    if (!ok && lane == 0 && atomicExch(const_cast<uint32_t*>(&bar->abort), 1u) == 0) dev::report(status, ST_TIMEOUT, blockIdx.x, 3, 0);
  } else if (warp >= FIRST_EPI_WARP) {
    // ------------------------------------------------------------------ epilogue (8 warps, both CTAs)
    const int quarter = warp & 3, strips = width / 32, per = (strips + 1) / 2;
    const int c_begin = ((warp - FIRST_EPI_WARP) >> 2) * per, c_end = c_begin + per < strips ? c_begin + per : strips;
    int acc = 0;
    uint32_t acc_phase = 0;
    bool ok = true;
    TileCoord t;
    for (int it = 0; ok && sched.get(it, &t); ++it) {
      if (!tc::mbar_wait(&bar->tmem_full[acc], acc_phase, abort)) { ok = false; break; }
      tc::tc_fence_after();
      const uint32_t taddr = tmem + (static_cast<uint32_t>(quarter * 32) << 16) + acc * 256;
      epi.tile_begin(t);
#pragma unroll 1
      for (int c = c_begin; c < c_end; ++c) {
        uint32_t r[32];
        tc::tmem_ld_32x32(taddr + c * 32, r);
        tc::tmem_ld_wait();
        epi.strip(t, quarter * 32 + lane, c * 32, r);
      }
      tc::tc_fence_before();
      __syncwarp();
      if (lane == 0) tc::mbar_arrive_remote(tc::mapa(tc::smem_u32(&bar->tmem_empty[acc]), 0));   // on the leader's barrier
      epi.tile_done(t, abort);
      if (++acc == 2) { acc = 0; acc_phase ^= 1; }
    }
    if (!ok && lane == 0 && atomicExch(const_cast<uint32_t*>(&bar->abort), 1u) == 0) dev::report(status, ST_TIMEOUT, blockIdx.x, 2, 0);
  }

  tc::tc_fence_before();
  __syncthreads();
  tc::cluster_sync();                 // the leader's MMAs no longer read the peer's shared memory
  if (warp == 1) {
    tc::tc_fence_after();
    tc::tmem_dealloc_pair(tmem, TMEM_COLS);
  }
}

}  // namespace gemmxp
}  // namespace pccl
