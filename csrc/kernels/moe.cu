// Expert-parallel MoE data movement fused with its arithmetic, plus the fp8 block quantisers.
//
//   dispatch   one pass per token: bf16 row -> e4m3 with one fp32 scale per 128 values (amax / 448),
//              staged in shared memory, then stored straight into the receive buffers of the ranks
//              that own the token's top-k experts (NVLink stores, 16 bytes per thread per target)
//   dequant    fp8 rows + scales -> bf16 rows for the grouped expert GEMM
//   combine    one pass per token: pull the top-k expert outputs from their ranks (up to 32
//              independent 16-byte NVLink loads in flight per thread), weight by the gate
//              probability, accumulate in fp32, write bf16
// Both communication kernels are persistent (one CTA per SM at most), open and close with a bounded
// peer barrier on per-CTA flags in the symmetric heap, and can emulate all ranks in one launch.
#include <cuda_bf16.h>
#include <cuda_fp8.h>

#include "gemm_api.h"
#include "gemm_epilogue.cuh"
#include "gemm_pipeline.cuh"
#include "gemm_pipeline2.cuh"
#include "launch.h"
#include "moe_api.h"
#include "prims.cuh"
#include "tensormap.h"

namespace pccl {

namespace {

using namespace dev;

__device__ __forceinline__ uint64_t* moe_flag(const World& W, int owner, int lane, int block, int src) {
  return reinterpret_cast<uint64_t*>(W.heap[owner] + W.flag_off) +
         ((static_cast<uint64_t>(lane) * kMaxBlocksPerColl + block) * kMaxRanks + src);
}

__device__ __forceinline__ bool moe_barrier(const MoeArgs& A, int me, uint64_t value, uint32_t* s_fail) {
  if (A.w.world == 1) return true;                // nobody to wait for, and no flags: the grid may have any size
  __syncthreads();
  if (threadIdx.x < static_cast<uint32_t>(A.w.world)) {
    const int p = threadIdx.x;
    __threadfence_system();
    st_release_sys(moe_flag(A.w, p, A.flag_lane, blockIdx.x, me), value);
    if (!wait_ge(moe_flag(A.w, me, A.flag_lane, blockIdx.x, p), value, A.spin_ns, nullptr)) {
      *s_fail = 1;
      report(A.status[A.nvirt > 1 ? me : 0], ST_TIMEOUT, blockIdx.x, static_cast<uint32_t>(p), static_cast<uint32_t>(value & 3));
    }
  }
  __syncthreads();
  return *s_fail == 0;
}

// Quantises 8 bf16 values with a given inverse scale into 8 e4m3 bytes.
__device__ __forceinline__ uint2 quant8(const float* f, float inv) {
  uint32_t w[2];
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    uint32_t lo = __nv_cvt_float2_to_fp8x2(make_float2(f[4 * h] * inv, f[4 * h + 1] * inv), __NV_SATFINITE, __NV_E4M3);
    uint32_t hi = __nv_cvt_float2_to_fp8x2(make_float2(f[4 * h + 2] * inv, f[4 * h + 3] * inv), __NV_SATFINITE, __NV_E4M3);
    w[h] = (lo & 0xffffu) | (hi << 16);
  }
  return make_uint2(w[0], w[1]);
}

// A token is a chain of dependent steps (load the row, block maxima, quantise, store), a few microseconds long whatever the
// bandwidth; one token at a time per SM leaves both HBM and NVLink idle most of the time.  So a CTA is up to kDispatchSubs (or kCombineSubs)
// groups of GT threads, each with its own staging row and its own named barrier, working on different tokens, and a group has the
// next token's row and routing in flight while it quantises and stores the current one.  GT = 64 threads to a group put the
// most tokens in flight and leave no thread idle in a row's last trip; with fewer tokens than groups a token's own chain
// counts, and it gets 256.  Times, us, 256 threads to a group -> 64, world of one: dispatch 4096 x 7168, top-8 36 -> 26.5, 4096 x 4096
// 60 -> 42 (scaled rows), 2001 x 2048, top-4 16.5 -> 10.5; combine 122 -> 115, 68 -> 64, 18.8 -> 13.4; gate gradients of 2001 x 2048
// 16.7 -> 11.0.  Loading the next vectors while these are added up was 109 us at 4096 x 7168, but 69 and 15.0 at the narrower ones.
template <int GT> constexpr int kDispatchSubs = GT == 64 ? 10 : 3;
template <int GT> constexpr int kCombineSubs = GT == 64 ? 8 : 2;
template <int GT> constexpr int kRowVecs = GT == 64 ? 8 : 4;       // vectors of 8 values per thread and chunk of a row
template <int GT> __device__ __forceinline__ void sub_sync(int sub) { asm volatile("bar.sync %0, %1;" ::"r"(sub + 1), "n"(GT) : "memory"); }
__host__ __device__ inline size_t dispatch_stage_bytes(int hidden) { return (static_cast<size_t>(hidden) + (hidden >> 7) * 4 + 15) / 16 * 16; }

// The routing of one token, one assignment per lane (lanes 0 .. topk - 1): destination rank (-1: dropped, or no assignment of
// this lane), row there, weight.
struct Assignment {
  int dest = -1, row = -1;
  float p = 0.f;
  __device__ __forceinline__ void fetch(const MoeArgs& A, int slot, int t, int lane, const float* weights) {
    dest = -1;
    row = -1;
    p = 0.f;
    if (t >= A.tokens || lane >= A.topk) return;
    const int at = t * A.topk + lane;
    const int e = A.expert_ids[slot][at];
    row = A.dst_rows[slot][at];
    if (weights) p = weights[at];
    if (e >= 0 && row >= 0) dest = e / A.experts_per_rank;
  }
};

template <int GT>
__device__ __forceinline__ void fetch_chunk(const __nv_bfloat16* x, int nvec, int v0, int tid, Vec16 (&r)[kRowVecs<GT>]) {
#pragma unroll
  for (int i = 0; i < kRowVecs<GT>; ++i) {
    const int v = v0 + tid + i * GT;
    if (v < nvec) r[i] = ld16(x + v * 8);
  }
}
// 16 consecutive lanes own one 128-value block, so the block amax is a half-warp shuffle reduction
template <int GT>
__device__ __forceinline__ void quant_chunk(const Vec16 (&r)[kRowVecs<GT>], int nvec, int v0, int tid, uint8_t* q, float* s) {
#pragma unroll
  for (int i = 0; i < kRowVecs<GT>; ++i) {
    const int v = v0 + tid + i * GT;
    if (v - (tid & 31) >= nvec) break;                  // warp-uniform for the shuffles
    float f[8];
    float amax = 0.f;
    if (v < nvec) {
      unpack<DT_BF16>(r[i], f);
#pragma unroll
      for (int k = 0; k < 8; ++k) amax = fmaxf(amax, fabsf(f[k]));
    }
#pragma unroll
    for (int o = 8; o > 0; o >>= 1) amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, o));
    const float scale = amax > 0.f ? amax * (1.0f / 448.0f) : 1.0f;
    if (v < nvec) {
      *reinterpret_cast<uint2*>(q + v * 8) = quant8(f, 1.0f / scale);
      if ((v & 15) == 0) s[v >> 4] = scale;
    }
  }
}

// One token after the other took 89 us at 4096 tokens x 7168, top-8, in a world of one; with the prefetch 37.
template <int GT>
__global__ void __launch_bounds__(GT * kDispatchSubs<GT>) moe_dispatch_kernel(const __grid_constant__ MoeArgs A) {
  extern __shared__ __align__(16) uint8_t dsm[];
  __shared__ uint32_t s_fail;
  if (threadIdx.x == 0) s_fail = 0;
  dev::pdl_launch();
  dev::pdl_wait();
  const int me = A.nvirt > 1 ? static_cast<int>(blockIdx.y) : A.rank;
  const int slot = A.nvirt > 1 ? me : 0;
  const int H = A.hidden, G = H >> 7, nvec = H >> 3;
  const int sub = threadIdx.x / GT, tid = threadIdx.x % GT, lane = threadIdx.x & 31, subs = blockDim.x / GT;
  uint8_t* q = dsm + sub * dispatch_stage_bytes(H);
  float* s = reinterpret_cast<float*>(q + H);
  if (!moe_barrier(A, me, 4 * A.epoch + 1, &s_fail)) return;
  const __nv_bfloat16* x = static_cast<const __nv_bfloat16*>(A.x[slot]);
  const int qvec = H >> 4, svec = (G + 3) >> 2;       // 16-byte vectors of payload / of scales
  const bool scaled = A.probs[slot] != nullptr;
  const bool dedupe = A.dedupe && A.alias_off && !scaled;      // scaled payloads differ per destination
  const float* weights = scaled ? A.probs[slot] : A.gate[slot];
  const int step = gridDim.x * subs;
  int t = blockIdx.x * subs + sub;
  Assignment next;
  Vec16 xv[kRowVecs<GT>];
  next.fetch(A, slot, t, lane, weights);
  if (t < A.tokens) fetch_chunk<GT>(x + static_cast<long long>(t) * H, nvec, 0, tid, xv);
  for (; t < A.tokens; t += step) {
    const Assignment a = next;
    sub_sync<GT>(sub);                                      // the previous token's stores have read the staging row
    quant_chunk<GT>(xv, nvec, 0, tid, q, s);
    for (int v0 = kRowVecs<GT> * GT; v0 < nvec; v0 += kRowVecs<GT> * GT) {          // rows longer than a chunk
      fetch_chunk<GT>(x + static_cast<long long>(t) * H, nvec, v0, tid, xv);
      quant_chunk<GT>(xv, nvec, v0, tid, q, s);
    }
    next.fetch(A, slot, t + step, lane, weights);
    if (t + step < A.tokens) fetch_chunk<GT>(x + static_cast<long long>(t + step) * H, nvec, 0, tid, xv);
    sub_sync<GT>(sub);
    // with de-duplication, the primary of an assignment is the token's first one to the same rank
    const uint32_t peers = __match_any_sync(0xffffffffu, a.dest);
    const int prim_l = dedupe ? __ffs(peers) - 1 : lane;
    for (int k = 0; k < A.topk; ++k) {
      const int dest = __shfl_sync(0xffffffffu, a.dest, k);
      if (dest < 0) continue;                           // dropped assignment (receive buffer full)
      const long long row = __shfl_sync(0xffffffffu, a.row, k);
      const int prim = __shfl_sync(0xffffffffu, prim_l, k);
      const int prim_row = __shfl_sync(0xffffffffu, a.row, prim);
      char* base = A.w.heap[dest];
      if (A.alias_off && tid == 0) reinterpret_cast<int*>(base + A.alias_off)[row] = prim_row;
      if (prim != k) continue;                          // the payload is already on its way to that rank
      if (dedupe && A.group_off) {
        // group record of this primary: the token's rows on that rank and their gate weights
        const int j = lane & 7;
        const bool member = __shfl_sync(0xffffffffu, a.dest, j) == dest;
        const int row_j = __shfl_sync(0xffffffffu, a.row, j);
        const float p_j = __shfl_sync(0xffffffffu, a.p, j);
        if (tid < 8) reinterpret_cast<uint32_t*>(base + A.group_off + row * 64)[tid] = member ? static_cast<uint32_t>(row_j) : 0xffffffffu;
        else if (tid < 16) reinterpret_cast<float*>(base + A.group_off + row * 64)[tid] = member ? p_j : 0.f;
      }
      char* dq = base + A.recv_q_off + row * H;
      char* ds = base + A.recv_s_off + row * G * 4;
      for (int v = tid; v < qvec; v += GT) st16(dq + v * 16, *reinterpret_cast<const Vec16*>(q + v * 16));
      // With gate weights attached, destination k receives p[t,k] * x[t] (the gradient of an expert's output row in
      // the backward pass): the e4m3 payload is the same for every destination, only the block scales are multiplied.
      const float p_k = __shfl_sync(0xffffffffu, a.p, k);
      const float pk = scaled ? p_k : 1.0f;
      for (int v = tid; v < svec; v += GT) {
        if ((G & 3) == 0 && !scaled) st16(ds + v * 16, *reinterpret_cast<const Vec16*>(reinterpret_cast<uint8_t*>(s) + v * 16));
        else for (int i = v * 4; i < min(G, v * 4 + 4); ++i) reinterpret_cast<float*>(ds)[i] = s[i] * pk;
      }
    }
  }
  moe_barrier(A, me, 4 * A.epoch + 2, &s_fail);
}

// Each group pulls a different token's rows, up to 16 vectors in flight per thread (what the registers of 512 threads allow).
template <int GT>
__global__ void __launch_bounds__(GT * kCombineSubs<GT>) moe_combine_kernel(const __grid_constant__ MoeArgs A) {
  __shared__ uint32_t s_fail;
  if (threadIdx.x == 0) s_fail = 0;
  dev::pdl_launch();
  dev::pdl_wait();
  const int me = A.nvirt > 1 ? static_cast<int>(blockIdx.y) : A.rank;
  const int slot = A.nvirt > 1 ? me : 0;
  const int H = A.hidden, nvec = H >> 3;
  const int sub = threadIdx.x / GT, tid = threadIdx.x % GT, lane = threadIdx.x & 31, subs = blockDim.x / GT;
  if (!moe_barrier(A, me, 4 * A.epoch + 1, &s_fail)) return;
  __nv_bfloat16* out = static_cast<__nv_bfloat16*>(A.out[slot]);
  const int step = gridDim.x * subs;
  int t = blockIdx.x * subs + sub;
  Assignment next;
  next.fetch(A, slot, t, lane, A.probs[slot]);
  for (; t < A.tokens; t += step) {
    const Assignment a = next;
    next.fetch(A, slot, t + step, lane, A.probs[slot]);       // in flight behind this token's rows
    const char* src_l = a.dest >= 0 ? A.w.heap[a.dest] + A.y_off + static_cast<long long>(a.row) * H * 2 : nullptr;
    float p_l = A.probs[slot] ? a.p : 1.0f;                 // without weights a plain sum
    const uint32_t peers = __match_any_sync(0xffffffffu, a.dest);
    if (A.dedupe && A.z_off && a.dest >= 0) {
      // one row per (token, rank): the first assignment to a rank stands for the token's whole group there; a group of two
      // or more has been summed (with its weights) into z on that rank, a group of one is still the plain expert output
      if (__ffs(peers) - 1 != lane) src_l = nullptr;
      else if (__popc(peers) > 1) {
        src_l = src_l - A.y_off + A.z_off;
        p_l = 1.0f;
      }
    }
    const char* src[8];
    float p[8];
#pragma unroll
    for (int k = 0; k < 8; ++k) {
      src[k] = reinterpret_cast<const char*>(__shfl_sync(0xffffffffu, reinterpret_cast<unsigned long long>(src_l), k));
      p[k] = __shfl_sync(0xffffffffu, p_l, k);
    }
    for (int v0 = tid; v0 < nvec; v0 += 2 * GT) {
      const int v1 = v0 + GT;
      Vec16 a[8], b[8];
#pragma unroll
      for (int k = 0; k < 8; ++k) {        // all loads first: up to 16 NVLink loads in flight per thread
        if (src[k]) {
          a[k] = ld16(src[k] + v0 * 16);
          if (v1 < nvec) b[k] = ld16(src[k] + v1 * 16);
        }
      }
      float acc0[8] = {0, 0, 0, 0, 0, 0, 0, 0}, acc1[8] = {0, 0, 0, 0, 0, 0, 0, 0};
#pragma unroll
      for (int k = 0; k < 8; ++k) {
        if (src[k]) {
          float f[8];
          unpack<DT_BF16>(a[k], f);
#pragma unroll
          for (int j = 0; j < 8; ++j) acc0[j] += p[k] * f[j];
          if (v1 < nvec) {
            unpack<DT_BF16>(b[k], f);
#pragma unroll
            for (int j = 0; j < 8; ++j) acc1[j] += p[k] * f[j];
          }
        }
      }
      st16(out + static_cast<long long>(t) * H + v0 * 8, pack<DT_BF16>(acc0));
      if (v1 < nvec) st16(out + static_cast<long long>(t) * H + v1 * 8, pack<DT_BF16>(acc1));
    }
  }
  moe_barrier(A, me, 4 * A.epoch + 2, &s_fail);
}

// dot[t,k] = <g[t], y[rank of expert (t,k)][dst_rows[t,k]]>: the gradient of the gate weight of an assignment, which is
// the upstream gradient of the token times the expert's output row.  The rows are pulled like in the combine.
template <int GT>
__global__ void __launch_bounds__(GT * kCombineSubs<GT>) moe_combine_dot_kernel(const __grid_constant__ MoeArgs A) {
  __shared__ uint32_t s_fail;
  __shared__ float part[kCombineSubs<GT>][GT / 32][8];
  if (threadIdx.x == 0) s_fail = 0;
  dev::pdl_launch();
  dev::pdl_wait();
  const int me = A.nvirt > 1 ? static_cast<int>(blockIdx.y) : A.rank;
  const int slot = A.nvirt > 1 ? me : 0;
  const int H = A.hidden, nvec = H >> 3;
  const int sub = threadIdx.x / GT, tid = threadIdx.x % GT, lane = threadIdx.x & 31, subs = blockDim.x / GT;
  if (!moe_barrier(A, me, 4 * A.epoch + 1, &s_fail)) return;
  const __nv_bfloat16* g = static_cast<const __nv_bfloat16*>(A.x[slot]);
  float* dot = static_cast<float*>(A.out[slot]);
  const int step = gridDim.x * subs;
  int t = blockIdx.x * subs + sub;
  Assignment next;
  next.fetch(A, slot, t, lane, nullptr);
  for (; t < A.tokens; t += step) {
    const Assignment a = next;
    next.fetch(A, slot, t + step, lane, nullptr);
    const char* src_l = a.dest >= 0 ? A.w.heap[a.dest] + A.y_off + static_cast<long long>(a.row) * H * 2 : nullptr;
    const char* src[8];
#pragma unroll
    for (int k = 0; k < 8; ++k)
      src[k] = reinterpret_cast<const char*>(__shfl_sync(0xffffffffu, reinterpret_cast<unsigned long long>(src_l), k));
    float acc[8] = {0, 0, 0, 0, 0, 0, 0, 0};
    for (int v = tid; v < nvec; v += GT) {
      Vec16 r[8];
#pragma unroll
      for (int k = 0; k < 8; ++k)
        if (src[k]) r[k] = ld16(src[k] + v * 16);
      float gf[8];
      unpack<DT_BF16>(ld16(g + static_cast<long long>(t) * H + v * 8), gf);
#pragma unroll
      for (int k = 0; k < 8; ++k) {
        if (src[k]) {
          float f[8];
          unpack<DT_BF16>(r[k], f);
#pragma unroll
          for (int j = 0; j < 8; ++j) acc[k] += gf[j] * f[j];
        }
      }
    }
#pragma unroll
    for (int k = 0; k < 8; ++k) {
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) acc[k] += __shfl_xor_sync(0xffffffffu, acc[k], o);
    }
    sub_sync<GT>(sub);
    if (lane == 0) {
#pragma unroll
      for (int k = 0; k < 8; ++k) part[sub][tid >> 5][k] = acc[k];
    }
    sub_sync<GT>(sub);
    if (tid < A.topk) {
      float sum = 0.f;
      for (int w = 0; w < GT / 32; ++w) sum += part[sub][w][tid];
      dot[t * A.topk + tid] = sum;
    }
  }
  moe_barrier(A, me, 4 * A.epoch + 2, &s_fail);
}

// One warp per row, eight values per lane and step (a warp stores 512 consecutive bytes), four steps in flight, the next row's
// alias fetched behind this row.  The e4m3 rows of a de-duplicated exchange come out of L2: 32768 rows of
// 7168 take 110 us, 470 MB stored at 4.3 TB/s (a CTA per row and half-filled second trips: 167).
__global__ void __launch_bounds__(256) moe_dequant_kernel(const uint8_t* q, const float* scales,
                                                          __nv_bfloat16* out, const int* n_rows,
                                                          int max_rows, int hidden, const int* alias) {
  dev::pdl_launch();
  dev::pdl_wait();
  const int rows = min(*n_rows, max_rows);
  const int nvec = hidden >> 3, G = hidden >> 7, lane = threadIdx.x & 31;
  const long long step = static_cast<long long>(gridDim.x) * 8;
  // a de-duplicated row: its payload sits in the token's primary row
  auto source = [&](long long r) { return alias && r < rows ? alias[r] : static_cast<int>(r); };
  long long r = static_cast<long long>(blockIdx.x) * 8 + (threadIdx.x >> 5);
  int src = source(r);
  for (; r < rows; r += step) {
    const long long from = src >= 0 && src < max_rows ? src : r;
    src = source(r + step);
    const uint8_t* qr = q + from * hidden + lane * 8;
    const float* sr = scales + from * G + (lane >> 4);
    __nv_bfloat16* o = out + r * hidden + lane * 8;
    for (int v = 0; v < nvec; v += 128) {
      uint2 x[4];
      float sc[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        if (v + i * 32 + lane < nvec) {
          x[i] = *reinterpret_cast<const uint2*>(qr + (v + i * 32) * 8);
          sc[i] = sr[(v + i * 32) >> 4];
        }
      }
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        if (v + i * 32 + lane < nvec) {
          float f[16];
          unpack<DT_FP8_E4M3>(Vec16{{x[i].x, x[i].y, 0u, 0u}}, f);
#pragma unroll
          for (int k = 0; k < 8; ++k) f[k] *= sc[i];
          st16(o + (v + i * 32) * 8, pack<DT_BF16>(f));
        }
      }
    }
  }
}

// Dispatch and conversion in one, for a world of one: nothing travels, so the rows that the experts read are written at once, without
// the e4m3 rows and scales in between (the values are those: quantised and converted back).  A warp takes 256 values of a token, 16 lanes a
// block of 128, with nothing kept from one to the next: the many short chains keep the memory busy better than longer ones (four vectors
// per thread 89 us, one 85), and a store is 512 consecutive bytes of one row.  The stores bound it.  Times, us, dispatch and conversion
// -> this (scaled by gate weights in brackets): 4096 x 7168, top-8 131 -> 85, 5.5 TB/s stored [183 -> 84]; 64 x 7168 10.8 -> 3.7;
// 2001 x 2048, top-4 14.1 -> 7.4 [17.4 -> 7.9]; 512 x 4096, top-2 15.0 -> 4.1; 128 x 1024, top-2 5.5 -> 2.5.
__global__ void __launch_bounds__(256) moe_expand_kernel(const __nv_bfloat16* x, const int* ids, const int* dst_rows, const float* probs, __nv_bfloat16* out,
                                                         int tokens, int topk, int hidden) {
  dev::pdl_launch();
  dev::pdl_wait();
  const int nvec = hidden >> 3, chunks = (nvec + 31) >> 5, lane = threadIdx.x & 31;
  const long long item = static_cast<long long>(blockIdx.x) * 8 + (threadIdx.x >> 5);
  const int t = static_cast<int>(item / chunks), v = static_cast<int>(item % chunks) * 32 + lane;
  if (t >= tokens) return;
  const bool in = v < nvec;                                 // the last chunk may be one block
  float f[16], amax = 0.f;
  if (in) unpack<DT_BF16>(ld16(x + static_cast<long long>(t) * hidden + v * 8), f);
  int row_l = -1;                                           // negative: dropped (receive buffer full), or no assignment of this lane
  float p_l = 1.f;
  if (lane < topk) {
    const long long at = static_cast<long long>(t) * topk + lane;
    if (ids[at] >= 0) row_l = dst_rows[at];
    if (probs) p_l = probs[at];
  }
  if (in) {
#pragma unroll
    for (int k = 0; k < 8; ++k) amax = fmaxf(amax, fabsf(f[k]));
  }
#pragma unroll
  for (int o = 8; o > 0; o >>= 1) amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, o));
  const float scale = amax > 0.f ? amax * (1.0f / 448.0f) : 1.0f;
  if (in) {
    const uint2 q = quant8(f, 1.0f / scale);
    unpack<DT_FP8_E4M3>(Vec16{{q.x, q.y, 0u, 0u}}, f);
  }
  Vec16 o;
#pragma unroll
  for (int k = 0; k < 8; ++k) {
    const int row = __shfl_sync(0xffffffffu, row_l, k);
    const float p = __shfl_sync(0xffffffffu, p_l, k);
    if (!in) continue;
    if (k == 0 || probs) {
      const float s = probs ? scale * p : scale;
      float g[8];
#pragma unroll
      for (int j = 0; j < 8; ++j) g[j] = f[j] * s;
      o = pack<DT_BF16>(g);
    }
    if (row >= 0) st16(out + static_cast<long long>(row) * hidden + v * 8, o);
  }
}

// z[r] = sum_j weight_j * y[row_j] over the group record of primary row r, for groups of two or more (a group of one stays in y
// and gets its weight in the combine).  Element-wise over the row, accumulated in fp32.
__global__ void __launch_bounds__(256) moe_reduce_groups_kernel(const __nv_bfloat16* y, __nv_bfloat16* z,
                                                                const int* alias, const uint32_t* groups,
                                                                const int* n_rows, int max_rows, int hidden) {
  dev::pdl_launch();
  dev::pdl_wait();
  const int rows = min(*n_rows, max_rows);
  const int nvec = hidden >> 3;
  for (long long r = blockIdx.x; r < rows; r += gridDim.x) {
    if (alias[r] != static_cast<int>(r)) continue;
    const uint32_t* g = groups + r * 16;
    int member[8];
    float w[8];
    int size = 0;
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      const int m = static_cast<int>(g[j]);
      member[j] = (m >= 0 && m < max_rows) ? m : -1;
      w[j] = __uint_as_float(g[8 + j]);
      size += member[j] >= 0;
    }
    if (size < 2) continue;
    for (int v = threadIdx.x; v < nvec; v += blockDim.x) {
      Vec16 a[8];
#pragma unroll
      for (int j = 0; j < 8; ++j)
        if (member[j] >= 0) a[j] = ld16(y + static_cast<long long>(member[j]) * hidden + v * 8);
      float acc[8] = {0, 0, 0, 0, 0, 0, 0, 0};
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        if (member[j] >= 0) {
          float f[8];
          unpack<DT_BF16>(a[j], f);
#pragma unroll
          for (int i = 0; i < 8; ++i) acc[i] += w[j] * f[i];
        }
      }
      st16(z + r * hidden + v * 8, pack<DT_BF16>(acc));
    }
  }
}

// Rows are whole 128-value blocks, so the matrix is one list of blocks, 16 lanes to each; PER loads in flight per thread: four,
// or one where that already puts the whole matrix in flight.  8192 x 8192: 61 -> 41 us (a CTA per row, staged in shared memory,
// before).
template <int PER>
__global__ void __launch_bounds__(256) quant_rows_kernel(const __nv_bfloat16* x, uint8_t* q,
                                                         float* scales, long long nvec) {
  dev::pdl_launch();
  dev::pdl_wait();
  constexpr int CHUNK = 256 * PER;
  for (long long v0 = static_cast<long long>(blockIdx.x) * CHUNK + threadIdx.x; v0 - (threadIdx.x & 31) < nvec; v0 += static_cast<long long>(gridDim.x) * CHUNK) {
    Vec16 in[PER];
#pragma unroll
    for (int j = 0; j < PER; ++j)
      if (v0 + j * 256 < nvec) in[j] = ld16(x + (v0 + j * 256) * 8);
#pragma unroll
    for (int j = 0; j < PER; ++j) {
      const long long v = v0 + j * 256;
      float f[8];
      float amax = 0.f;
      if (v < nvec) {
        unpack<DT_BF16>(in[j], f);
#pragma unroll
        for (int k = 0; k < 8; ++k) amax = fmaxf(amax, fabsf(f[k]));
      }
#pragma unroll
      for (int o = 8; o > 0; o >>= 1) amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, o));
      const float scale = amax > 0.f ? amax * (1.0f / 448.0f) : 1.0f;
      if (v < nvec) {
        *reinterpret_cast<uint2*>(q + v * 8) = quant8(f, 1.0f / scale);
        if ((v & 15) == 0) scales[v >> 4] = scale;
      }
    }
  }
}

// one CTA per 128 x 128 block of a weight matrix
__global__ void __launch_bounds__(256) quant_blocks_kernel(const __nv_bfloat16* __restrict__ w, uint8_t* __restrict__ q,
                                                           float* __restrict__ scales, int rows, int cols) {
  __shared__ float red[8];
  const int bc = blockIdx.x, br = blockIdx.y;
  const __nv_bfloat16* base = w + static_cast<long long>(br) * 128 * cols + bc * 128;
  float f[8][8];
  float amax = 0.f;
  // 128 x 128 values = 2048 vectors of 8; 256 threads take 8 each: thread -> (row group, vector in row)
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    const int idx = threadIdx.x + i * 256, r = idx >> 4, v = idx & 15;
    unpack<DT_BF16>(ld16(base + static_cast<long long>(r) * cols + v * 8), f[i]);
#pragma unroll
    for (int k = 0; k < 8; ++k) amax = fmaxf(amax, fabsf(f[i][k]));
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, o));
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = amax;
  __syncthreads();
  amax = red[0];
#pragma unroll
  for (int i = 1; i < 8; ++i) amax = fmaxf(amax, red[i]);
  const float scale = amax > 0.f ? amax * (1.0f / 448.0f) : 1.0f;
  if (threadIdx.x == 0) scales[br * (cols >> 7) + bc] = scale;
  const float inv = 1.0f / scale;
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    const int idx = threadIdx.x + i * 256, r = idx >> 4, v = idx & 15;
    *reinterpret_cast<uint2*>(q + (static_cast<long long>(br) * 128 + r) * cols + bc * 128 + v * 8) = quant8(f[i], inv);
  }
}

// ---------------------------------------------------------------------------------------------
// grouped GEMM on the tcgen05 pipeline
// ---------------------------------------------------------------------------------------------
using namespace gemm;

// Both schedulers walk the concatenated per-group tile lists.  A role asks for its tiles in increasing order, so each keeps a
// cursor (group, tiles before it) instead of scanning the groups from the start for every tile: the scan is a chain of
// dependent loads, and the MMA warp's share of it would sit between two tiles with the tensor cores idle.
struct GroupedSched {
  const int* row_off;    // groups + 1
  int groups, tiles_n, first, stride;
  int tile_rows;
  mutable int cur_g = 0;
  mutable long long cur_base = 0;
  // Tile `idx` of the concatenated per-group tile lists -> (group, m-tile inside group, n-tile).
  __device__ __forceinline__ bool get(int it, TileCoord* t) const {
    const long long idx = first + static_cast<long long>(it) * stride;
    while (cur_g < groups) {
      const int rows = row_off[cur_g + 1] - row_off[cur_g];
      const int tm = (rows + tile_rows - 1) / tile_rows;
      const long long tiles = static_cast<long long>(tm) * tiles_n;
      if (idx - cur_base < tiles) {
        const int local = static_cast<int>(idx - cur_base);
        t->m = local % tm;
        t->n = local / tm;
        t->extra = cur_g;
        return true;
      }
      cur_base += tiles;
      ++cur_g;
    }
    return false;
  }
};

struct GroupedEpi {
  __nv_bfloat16* D;
  long long ldd;
  const int* row_off;
  int N;
  uint32_t flags;
  __device__ __forceinline__ int a_row0(const TileCoord& t) const { return row_off[t.extra] + t.m * BM; }
  __device__ __forceinline__ int b_row0(const TileCoord& t) const { return t.extra * N + t.n * BN; }
  __device__ __forceinline__ void attach_smem(uint8_t*) {}
  __device__ __forceinline__ void tile_begin(const TileCoord&) {}
  __device__ __forceinline__ void tile_done(const TileCoord&, const volatile uint32_t*) {}
  __device__ __forceinline__ void strip(const TileCoord& t, int row_in_tile, int col_in_tile, uint32_t* r) {
    const int row = row_off[t.extra] + t.m * BM + row_in_tile;
    const int col = t.n * BN + col_in_tile;
    if (row >= row_off[t.extra + 1] || col >= N) return;     // rows past the group's end belong to the next group
    float v[32];
#pragma unroll
    for (int i = 0; i < 32; ++i) v[i] = __uint_as_float(r[i]);
    if (flags & GEMM_GELU_INPLACE) {
#pragma unroll
      for (int i = 0; i < 32; ++i) v[i] = gelu_tanh(v[i]);
    }
    __nv_bfloat16* d = D + static_cast<long long>(row) * ldd + col;
    if (col + 32 <= N && reinterpret_cast<uintptr_t>(D) % 16 == 0) {
#pragma unroll
      for (int i = 0; i < 32; i += 8) st16(d + i, pack<DT_BF16>(v + i));
    } else {
#pragma unroll
      for (int i = 0; i < 32; ++i)
        if (col + i < N) d[i] = __float2bfloat16_rn(v[i]);
    }
  }
};

__global__ void __launch_bounds__(NUM_THREADS, 1)
gemm_grouped_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB, GroupedEpi epi, int groups, int K,
                    uint32_t* status) {
  GroupedSched sched{epi.row_off, groups, (epi.N + BN - 1) / BN, static_cast<int>(blockIdx.x), static_cast<int>(gridDim.x), BM};
  NoGate gate;
  run<false, false>(&tmA, &tmB, K, sched, gate, epi, status);
}

// The same product with the operands exchanged: the weights of a group are the M side of the tile (256 output features; the
// last tile of a group may reach into the next group's weights, its surplus rows are not stored) and the group's rows are the
// N side, whose extent the MMA instruction takes per tile in steps of 16.  A group of 520 rows then costs 2 + 8/256 tiles of
// tensor time per weight tile, where the row-major form above pays for 3: with a few hundred rows per expert that is a fifth of
// the whole product.  The accumulator arrives transposed (lane = output feature, column = row of the group), so a warp stores
// 32 consecutive features of one row per instruction.  The row-major form is left with what the 8-byte stores of this one cannot
// write: feature counts that are no multiple of four and outputs off the 8-byte boundaries.
struct RaggedSched {
  const int* row_off;
  int groups, tiles_f, first, stride;        // tiles_f = ceil(N / 256) weight tiles per group
  mutable int cur_g = 0;
  mutable long long cur_base = 0;
  __device__ __forceinline__ bool get(int it, TileCoord* t) const {
    const long long idx = first + static_cast<long long>(it) * stride;
    while (cur_g < groups) {
      const int rows = row_off[cur_g + 1] - row_off[cur_g];
      const int tr = (rows + 255) / 256;
      const long long tiles = static_cast<long long>(tr) * tiles_f;
      if (idx - cur_base < tiles) {
        const int local = static_cast<int>(idx - cur_base);
        t->m = local / tr;                     // weight tile; the row tiles of one weight tile are neighbours in the list
        t->n = local % tr;
        t->extra = cur_g;
        return true;
      }
      cur_base += tiles;
      ++cur_g;
    }
    return false;
  }
};

// The epilogue of the exchanged form, with the element-wise work of the expert MLP in it:
//   GEMM_GELU_INPLACE  D = gelu(acc)                      (serving)
//   GEMM_GELU          D = acc, D2 = gelu(acc)            (training: the pre-activation is kept for the backward pass)
//   GEMM_DGELU         D = acc * gelu'(D2)                (backward, D2 = the pre-activation)
// W_MN: the weights of a group are stored [K, N] (the backward pass multiplies by the transposed weights of the forward pass).
template <bool W_MN>
struct RaggedEpi {
  static constexpr bool kVarN = true;
  __nv_bfloat16* D;
  __nv_bfloat16* D2;
  long long ldd;
  const int* row_off;
  int N;             // output features per group
  int K;
  uint32_t flags;
  int cta;
  __device__ __forceinline__ int tile_n(const TileCoord& t) const {
    const int left = row_off[t.extra + 1] - row_off[t.extra] - t.n * 256;
    return left >= 256 ? 256 : ((left + 15) & ~15);
  }
  // A operand: this CTA's 128 weight rows; B operand: this CTA's half of the tile's rows
  // descriptor whose box holds 128 >> b_box rows: the smallest that covers this CTA's tile_n / 2 rows
  __device__ __forceinline__ int b_box(const TileCoord& t) const {
    const int half = tile_n(t) >> 1;
    return half > 64 ? 0 : half > 32 ? 1 : half > 16 ? 2 : half > 8 ? 3 : 4;
  }
  __device__ __forceinline__ int a_row0(const TileCoord& t) const { return (W_MN ? 0 : t.extra * N) + t.m * 256 + cta * 128; }
  __device__ __forceinline__ int a_k0(const TileCoord& t) const { return W_MN ? t.extra * K : 0; }
  __device__ __forceinline__ int b_row0(const TileCoord& t) const { return row_off[t.extra] + t.n * 256 + cta * (tile_n(t) >> 1); }
  __device__ __forceinline__ void attach_smem(uint8_t*) {}
  int tile_row0 = 0, group_end = 0;         // epilogue warps: the tile's first row and the group's end, read once per tile
  __device__ __forceinline__ void tile_begin(const TileCoord& t) {
    tile_row0 = row_off[t.extra] + t.n * 256;
    group_end = row_off[t.extra + 1];
  }
  __device__ __forceinline__ void tile_done(const TileCoord&, const volatile uint32_t*) {}

  // The lane holds 32 rows of ONE feature; its neighbours hold the next features of the same rows.  Two exchange steps
  // (lane ^ 1, lane ^ 2) regroup that into 4 consecutive features of one row per lane, so a strip leaves as 8 stores of 8 bytes
  // per lane instead of 32 of 2: lanes 4q..4q+3 then cover rows 4j+0..3 of features 4q..4q+3.  `at` is row 0 of the strip at the
  // lane's four features, null where those lie past N.
  static __device__ __forceinline__ void put(__nv_bfloat16* at, long long ldd, int lane, int n_valid, const float* v) {
    const bool odd1 = lane & 1, odd2 = lane & 2;
    uint32_t p[16];
#pragma unroll
    for (int j = 0; j < 16; ++j) {
      const float a = v[2 * j], b = v[2 * j + 1];
      const float got = __shfl_xor_sync(0xffffffffu, odd1 ? a : b, 1);
      // even lane: row 2j, features (f, f+1) = (own a, neighbour's a); odd lane: row 2j+1, features (f-1, f) = (neighbour's b, own b)
      const __nv_bfloat162 x = odd1 ? __floats2bfloat162_rn(got, b) : __floats2bfloat162_rn(a, got);
      p[j] = *reinterpret_cast<const uint32_t*>(&x);
    }
#pragma unroll
    for (int m = 0; m < 8; ++m) {
      const uint32_t got = __shfl_xor_sync(0xffffffffu, odd2 ? p[2 * m] : p[2 * m + 1], 2);
      // bit 1 clear: keeps pair-row 2m, features +0..1 own, +2..3 from lane ^ 2; bit 1 set: keeps pair-row 2m+1
      const uint2 out = odd2 ? make_uint2(got, p[2 * m + 1]) : make_uint2(p[2 * m], got);
      const int row = 2 * (2 * m + (odd2 ? 1 : 0)) + (odd1 ? 1 : 0);
      if (at && row < n_valid) *reinterpret_cast<uint2*>(at + row * ldd) = out;
    }
  }
  // The same exchange the other way round: 8 loads of 8 bytes, then lane ^ 2, lane ^ 1; rows past n_valid read as zero.
  static __device__ __forceinline__ void get(const __nv_bfloat16* at, long long ldd, int lane, int n_valid, float* v) {
    const bool odd1 = lane & 1, odd2 = lane & 2;
    uint2 in[8];
#pragma unroll
    for (int m = 0; m < 8; ++m) {
      const int row = 2 * (2 * m + (odd2 ? 1 : 0)) + (odd1 ? 1 : 0);
      in[m] = at && row < n_valid ? *reinterpret_cast<const uint2*>(at + row * ldd) : make_uint2(0u, 0u);
    }
#pragma unroll
    for (int m = 0; m < 8; ++m) {
      const uint32_t got = __shfl_xor_sync(0xffffffffu, odd2 ? in[m].x : in[m].y, 2);
      const uint32_t p[2] = {odd2 ? got : in[m].x, odd2 ? in[m].y : got};
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        // p = (low: feature of the even lane, high: feature of the odd lane) of row 2j (even lane) or 2j+1 (odd lane)
        const uint32_t other = __shfl_xor_sync(0xffffffffu, odd1 ? p[i] << 16 : p[i] & 0xffff0000u, 1);
        const int j = 2 * m + i;
        v[2 * j] = __uint_as_float(odd1 ? other : p[i] << 16);
        v[2 * j + 1] = __uint_as_float(odd1 ? p[i] & 0xffff0000u : other);
      }
    }
  }
  __device__ __forceinline__ void strip(const TileCoord& t, int feat_in_cta, int col0, uint32_t* r) {
    const int lane = feat_in_cta & 31;
    const int feat4 = t.m * 256 + cta * 128 + (feat_in_cta & ~3);
    const int row0 = tile_row0 + col0;
    const int n_valid = group_end - row0;                     // rows of this strip that belong to the group (may exceed 32)
    const long long off = row0 * ldd + feat4;
    const bool in = feat4 < N;                                // N % 4 == 0
    float v[32];
#pragma unroll
    for (int i = 0; i < 32; ++i) v[i] = __uint_as_float(r[i]);
    if (flags & GEMM_DGELU) {
      float pre[32];
      get(in ? D2 + off : nullptr, ldd, lane, n_valid, pre);
#pragma unroll
      for (int i = 0; i < 32; ++i) v[i] *= dgelu_logistic(pre[i]);
    }
    if (flags & GEMM_GELU_INPLACE) {
#pragma unroll
      for (int i = 0; i < 32; ++i) v[i] = gelu_tanh(v[i]);
    }
    put(in ? D + off : nullptr, ldd, lane, n_valid, v);
    if (flags & GEMM_GELU) {
#pragma unroll
      for (int i = 0; i < 32; ++i) v[i] = gelu_logistic(v[i]);
      put(in ? D2 + off : nullptr, ldd, lane, n_valid, v);
    }
  }
};

struct RaggedMaps { CUtensorMap x[5]; };     // boxes of 128, 64, 32, 16, 8 rows

template <bool W_MN>
__global__ void __launch_bounds__(gemm2::NUM_THREADS_WIDE, 1)
gemm_grouped_ragged_kernel(const __grid_constant__ CUtensorMap tmW, const __grid_constant__ RaggedMaps tmX, RaggedEpi<W_MN> epi, int groups,
                           int K, uint32_t* status) {
  RaggedSched sched{epi.row_off, groups, (epi.N + 255) / 256, static_cast<int>(blockIdx.x >> 1), static_cast<int>(gridDim.x >> 1)};
  NoGate gate;
  epi.cta = static_cast<int>(tc::cluster_ctarank());
  gemm2::run<W_MN, false, RaggedSched, NoGate, RaggedEpi<W_MN>, gemm2::STAGES, 1, false, 8>(&tmW, tmX.x, K, sched, gate, epi, status);
}

// ---------------------------------------------------------------------------------------------
// grouped weight gradients
// ---------------------------------------------------------------------------------------------
// D_q[g] = A_q[rows of g]^T * B_q[rows of g] for every group g and the two projections q of the expert MLP as one tile list:
// M_q x N_q outputs per group, reduced over the group's rows, whose number only the device knows.  Both operands are read
// where they lie (MN-major).  The reduction of a group ends in the middle of a k-block as a rule, and what follows in memory
// are the next group's rows; so every (group, operand) has a descriptor of its own whose outer extent is the group's end, and
// TMA fills the rest of the block with zeros.  The descriptors are made on the device from four templates, one warp each.
// A group without rows gets zeros.
struct WgradTemplates { CUtensorMap m[4]; };           // A_0, B_0, A_1, B_1

__global__ void __launch_bounds__(128) wgrad_maps_kernel(const __grid_constant__ WgradTemplates tmpl, const int* __restrict__ row_off,
                                                         int max_rows, CUtensorMap* __restrict__ maps) {
  __shared__ __align__(128) CUtensorMap stage[4];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, g = blockIdx.x;
  reinterpret_cast<uint32_t*>(&stage[warp])[lane] = reinterpret_cast<const uint32_t*>(&tmpl.m[warp])[lane];
  __syncwarp();
  if (lane == 0) tc::tensormap_set_outer(&stage[warp], static_cast<uint32_t>(max(1, min(row_off[g + 1], max_rows))));     // never past the operands
  __syncwarp();
  tc::tensormap_publish(maps + g * 4 + warp, &stage[warp]);
}

struct WgradSched {
  int tiles_m[2], tiles_n[2], groups, first, stride;
  __device__ __forceinline__ bool get(int it, TileCoord* t) const {
    const long long idx = first + static_cast<long long>(it) * stride;
    const int n0 = tiles_m[0] * tiles_n[0], per = n0 + tiles_m[1] * tiles_n[1];
    const int g = static_cast<int>(idx / per);
    if (g >= groups) return false;
    int r = static_cast<int>(idx - static_cast<long long>(g) * per);
    const int q = r >= n0 ? 1 : 0;
    if (q) r -= n0;
    const int tm = q ? tiles_m[1] : tiles_m[0];         // no variable index: the array would live in local memory
    t->m = r % tm;
    t->n = r / tm;
    t->extra = g * 2 + q;
    return true;
  }
};

struct WgradEpi {
  static constexpr bool kRaggedK = true;
  StoreEpi e[2];               // D: group 0
  const int* row_off;
  const CUtensorMap* maps;     // [groups][4]
  int cta;
  __device__ __forceinline__ int k_begin(const TileCoord& t) const { return row_off[t.extra >> 1]; }
  __device__ __forceinline__ int k_blocks(const TileCoord& t) const {
    return (row_off[(t.extra >> 1) + 1] - row_off[t.extra >> 1] + gemm2::BK - 1) / gemm2::BK;
  }
  __device__ __forceinline__ const CUtensorMap* a_map(const TileCoord& t) const { return maps + t.extra * 2; }
  __device__ __forceinline__ const CUtensorMap* b_map(const TileCoord& t) const { return maps + t.extra * 2 + 1; }
  __device__ __forceinline__ int a_row0(const TileCoord& t) const { return t.m * 256 + cta * 128; }
  __device__ __forceinline__ int b_row0(const TileCoord& t) const { return t.n * 256 + cta * 128; }
  __device__ __forceinline__ void attach_smem(uint8_t*) {}
  __device__ __forceinline__ void attach_patch(uint8_t* p) { e[0].attach_patch(p); e[1].attach_patch(p); }
  // The tile's problem is picked once per tile, value by value: indexed with a variable the two would live in local memory, and every
  // strip of these short tiles (four k-blocks at 250 rows per group) would read its problem and the group's rows from there and from
  // global memory: 140 -> 99 us at 2001 tokens, 32 experts, top-4, 2048 x 1024.
  StoreEpi cur;
  bool empty = false;
  __device__ __forceinline__ void tile_begin(const TileCoord& t) {
    const int g = t.extra >> 1;
    cur = e[0];
    if (t.extra & 1) cur = e[1];
    cur.D = static_cast<__nv_bfloat16*>(cur.D) + static_cast<long long>(g) * cur.M * cur.ldd;
    empty = row_off[g + 1] == row_off[g];
  }
  __device__ __forceinline__ void tile_done(const TileCoord&, const volatile uint32_t*) {}
  __device__ __forceinline__ void strip(const TileCoord& t, int row, int col, uint32_t* r) {
    if (empty) {
#pragma unroll
      for (int i = 0; i < 32; ++i) r[i] = 0u;          // nothing was accumulated
    }
    cur.strip(TileCoord{t.m * 2 + cta, t.n, 0}, row, col, r);
  }
};

__global__ void __launch_bounds__(gemm2::NUM_THREADS_WIDE, 1) gemm_grouped_wgrad_kernel(WgradEpi epi, int groups, uint32_t* status) {
  WgradSched sched{{(epi.e[0].M + 255) / 256, (epi.e[1].M + 255) / 256}, {(epi.e[0].N + 255) / 256, (epi.e[1].N + 255) / 256}, groups,
                   static_cast<int>(blockIdx.x >> 1), static_cast<int>(gridDim.x >> 1)};
  NoGate gate;
  epi.cta = static_cast<int>(tc::cluster_ctarank());
  gemm2::run<true, true, WgradSched, NoGate, WgradEpi, gemm2::STAGES, 1, false, 8>(nullptr, nullptr, gemm2::BK, sched, gate, epi, status);
}

// ---------------------------------------------------------------------------------------------
// routing and placement
// ---------------------------------------------------------------------------------------------
template <int PER_LANE>
__device__ __forceinline__ void route_token(const float* logits, int* ids, float* probs, int* pos,
                                            int* cnt, int t, int experts, int topk, int lane) {
  float v[PER_LANE];
  float mx = -INFINITY;
#pragma unroll
  for (int j = 0; j < PER_LANE; ++j) {
    const int e = j * 32 + lane;
    v[j] = e < experts ? logits[static_cast<long long>(t) * experts + e] : -INFINITY;
    mx = fmaxf(mx, v[j]);
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
  float sum = 0.f;
#pragma unroll
  for (int j = 0; j < PER_LANE; ++j) {
    const float p = __expf(v[j] - mx);
    sum += p;
    v[j] = j * 32 + lane < experts ? p : -2.f;       // the padding is never taken, also where all logits left are NaN
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
  const float inv = 1.f / sum;
  for (int k = 0; k < topk; ++k) {
    float best = -1.f;
    int bi = 0;
#pragma unroll
    for (int j = 0; j < PER_LANE; ++j)
      if (v[j] > best) { best = v[j]; bi = j * 32 + lane; }
    // warp arg-max; ties go to the lower expert id (what a stable top-k returns)
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      const float ob = __shfl_xor_sync(0xffffffffu, best, o);
      const int oi = __shfl_xor_sync(0xffffffffu, bi, o);
      if (ob > best || (ob == best && oi < bi)) { best = ob; bi = oi; }
    }
    if ((bi & 31) == lane) {
#pragma unroll
      for (int j = 0; j < PER_LANE; ++j)
        if (j == (bi >> 5)) v[j] = -2.f;       // taken
      ids[t * topk + k] = bi;
      probs[t * topk + k] = best * inv;
      pos[t * topk + k] = atomicAdd(cnt + bi, 1);
    }
  }
}

// One warp per token.  An assignment's place among those of its expert comes from counters.  SHARED: a block of up to 32 tokens
// counts in shared memory and draws its share of each expert's rows with one global atomic; with an atomic per assignment
// 4096 tokens, top-8, over 8 / 32 / 64 / 128 / 256 experts take 28 / 27 / 27 / 18 / 19 us instead of 12 / 11 / 12 / 13 / 15, because
// they queue up behind one another.  Where few assignments meet (64 tokens over 256 experts) or a block would walk hundreds of
// counters for its handful of assignments, the atomic per assignment is the faster: 10 against 12 us there, 18 against 19 at
// 4096 x 512, 12 against 20 at 64 x 1024.
template <int PER_LANE, bool SHARED>
__global__ void __launch_bounds__(SHARED ? 1024 : 256) moe_route_kernel(const float* logits, int* ids, float* probs, int* pos, int* counts, int tokens,
                                                                        int experts, int topk) {
  extern __shared__ int cnt[];             // SHARED: [experts] assignments of this block, then the first place of the block
  const int lane = threadIdx.x & 31;
  const int t0 = blockIdx.x * (blockDim.x >> 5), t = t0 + (threadIdx.x >> 5);
  if (SHARED)
    for (int e = threadIdx.x; e < experts; e += blockDim.x) cnt[e] = 0;
  dev::pdl_launch();
  dev::pdl_wait();
  if (SHARED) __syncthreads();
  if (t < tokens) route_token<PER_LANE>(logits, ids, probs, pos, SHARED ? cnt : counts, t, experts, topk, lane);
  if (!SHARED) return;
  __syncthreads();
  for (int e = threadIdx.x; e < experts; e += blockDim.x)
    if (cnt[e]) cnt[e] = atomicAdd(counts + e, cnt[e]);
  __syncthreads();
  const int end = min(tokens, t0 + static_cast<int>(blockDim.x >> 5)) * topk;
  for (int i = t0 * topk + threadIdx.x; i < end; i += blockDim.x) pos[i] += cnt[ids[i]];     // both written by this block above
}

__global__ void __launch_bounds__(256) moe_plan_kernel(const int* counts_all, const int* ids, const int* pos,
                                                       int* rows, int* row_off, int world, int rank, int experts,
                                                       int tokens, int topk, int cap) {
  extern __shared__ int first[];           // [experts + 1] rows of the experts before e, over all ranks of the world
  __shared__ int warp_sum[8];
  dev::pdl_launch();
  dev::pdl_wait();
  const int epr = experts / world, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int per = (experts + 255) / 256, e0 = threadIdx.x * per, e1 = min(experts, e0 + per);
  int mine = 0;
  for (int e = e0; e < e1; ++e) {
    int n = 0;
    for (int r = 0; r < world; ++r) n += counts_all[r * experts + e];
    first[e] = n;
    mine += n;
  }
  int incl = mine;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int x = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= o) incl += x;
  }
  if (lane == 31) warp_sum[warp] = incl;
  __syncthreads();
  int at = incl - mine;
  for (int w = 0; w < warp; ++w) at += warp_sum[w];
  for (int e = e0; e < e1; ++e) {
    const int n = first[e];
    first[e] = at;
    at += n;
  }
  if (threadIdx.x == 255) first[experts] = at;         // the last thread's running sum is the total
  __syncthreads();
  if (blockIdx.x == 0)
    for (int i = threadIdx.x; i <= epr; i += blockDim.x) row_off[i] = min(first[rank * epr + i] - first[rank * epr], cap);
  const int total = tokens * topk;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < total; i += gridDim.x * blockDim.x) {
    const int e = ids[i];
    int row = first[e] - first[e / epr * epr] + pos[i];
    for (int r = 0; r < rank; ++r) row += counts_all[r * experts + e];       // lower ranks come first inside the expert's segment
    rows[i] = row < cap ? row : -1;
  }
}

// Gradient of the routing logits of one token per warp: with p = softmax(logits) over all experts and d the gradients of the weights
// of the experts taken (zero for the others), p .* (d - <p, d>).  The exponentials are taken in fp64, a few per lane: the fast
// ones of this file are good to 1e-6 only.  One launch of 3 us for eight of tensor operations (25 us, 2001 tokens, 32 experts).
template <int PER_LANE>
__global__ void __launch_bounds__(256) moe_route_backward_kernel(const float* logits, const int* ids, const float* dprobs, float* dlogits, int tokens,
                                                                 int experts, int topk) {
  dev::pdl_launch();
  dev::pdl_wait();
  const int lane = threadIdx.x & 31, t = blockIdx.x * 8 + (threadIdx.x >> 5);
  if (t >= tokens) return;
  float p[PER_LANE], d[PER_LANE];
  float mx = -INFINITY;
#pragma unroll
  for (int j = 0; j < PER_LANE; ++j) {
    const int e = j * 32 + lane;
    p[j] = e < experts ? ld_f32(logits + static_cast<long long>(t) * experts + e) : -INFINITY;
    d[j] = 0.f;
    mx = fmaxf(mx, p[j]);
  }
  for (int k = 0; k < topk; ++k) {
    const int e = static_cast<int>(ld_u32(ids + t * topk + k));
    const float g = ld_f32(dprobs + t * topk + k);
#pragma unroll
    for (int j = 0; j < PER_LANE; ++j)
      if (j * 32 + lane == e) d[j] = g;
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
  float sum = 0.f;
#pragma unroll
  for (int j = 0; j < PER_LANE; ++j) {
    p[j] = j * 32 + lane < experts ? static_cast<float>(exp(static_cast<double>(p[j]) - mx)) : 0.f;
    sum += p[j];
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
  float dot = 0.f;
#pragma unroll
  for (int j = 0; j < PER_LANE; ++j) {
    p[j] = __fdiv_rn(p[j], sum);
    dot += p[j] * d[j];
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) dot += __shfl_xor_sync(0xffffffffu, dot, o);
#pragma unroll
  for (int j = 0; j < PER_LANE; ++j) {
    const int e = j * 32 + lane;
    if (e < experts) dlogits[static_cast<long long>(t) * experts + e] = p[j] * (d[j] - dot);
  }
}

template <typename K>
int coop(K kernel, const MoeArgs& a, int blocks, size_t smem, cudaStream_t stream, int threads, int subs, int ctas_per_sm) {
  if (blocks < 1) blocks = 1;
  // A world of one has no barrier, so neither flags nor co-residency limit the grid: `ctas_per_sm` times the blocks asked for,
  // no more than there are tokens.
  const int groups = (a.tokens + subs - 1) / subs;
  const int world_of_one = groups < 1 ? 1 : groups < blocks * ctas_per_sm ? groups : blocks * ctas_per_sm;
  if (blocks > kMaxBlocksPerColl) blocks = kMaxBlocksPerColl;
  if (a.topk > 8 || a.hidden % 128 || a.flag_lane < 0 || a.flag_lane >= 8) return static_cast<int>(cudaErrorInvalidValue);
  if (a.w.world == 1) return static_cast<int>(launchOverlapped(kernel, dim3(world_of_one), dim3(threads), smem, stream, 1, a));
  dim3 grid(blocks, a.nvirt > 1 ? a.nvirt : 1), block(threads);
  void* args[] = {const_cast<MoeArgs*>(&a)};
  return static_cast<int>(cudaLaunchCooperativeKernel(reinterpret_cast<void*>(kernel), grid, block, args, smem, stream));
}

template <int GT>
int dispatchGroups(const MoeArgs& a, int blocks, cudaStream_t stream) {
  int subs = kDispatchSubs<GT>;                   // fewer where the staging rows of very long tokens would not fit
  while (subs > 1 && subs * dispatch_stage_bytes(a.hidden) > 200 * 1024) --subs;
  const size_t smem = subs * dispatch_stage_bytes(a.hidden);
  static size_t smem_set = 0;
  if (smem > 48 * 1024 && smem > smem_set) {
    cudaError_t e = cudaFuncSetAttribute(moe_dispatch_kernel<GT>, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(smem));
    if (e != cudaSuccess) return static_cast<int>(e);
    smem_set = smem;
  }
  return coop(moe_dispatch_kernel<GT>, a, blocks, smem, stream, GT * subs, subs, 1);
}

}  // namespace

// Groups of 64 threads are taken in a world of one, from two tokens on for every group of 256 that the blocks hold (64 tokens x 7168 stay as
// they were, 700 x 1024 takes 5.6 -> 3.6 us in the combine).  Between ranks, where rows cross NVLink and barriers frame the kernel, groups
// of 256 are what was measured.
int moeGroupThreads(bool dispatch, int tokens, int blocks, int world) {
  return world == 1 && tokens >= 2 * (dispatch ? kDispatchSubs<256> : kCombineSubs<256>) * (blocks < 1 ? 1 : blocks) ? 64 : 256;
}

int launchMoeDispatch(const MoeArgs& a, int blocks, cudaStream_t stream) {
  return moeGroupThreads(true, a.tokens, blocks, a.w.world) == 64 ? dispatchGroups<64>(a, blocks, stream) : dispatchGroups<256>(a, blocks, stream);
}

int launchMoeCombine(const MoeArgs& a, int blocks, cudaStream_t stream) {
  return moeGroupThreads(false, a.tokens, blocks, a.w.world) == 64
             ? coop(moe_combine_kernel<64>, a, blocks, 0, stream, 64 * kCombineSubs<64>, kCombineSubs<64>, 1)
             : coop(moe_combine_kernel<256>, a, blocks, 0, stream, 256 * kCombineSubs<256>, kCombineSubs<256>, 1);
}
int launchMoeCombineDot(const MoeArgs& a, int blocks, cudaStream_t stream) {
  return moeGroupThreads(false, a.tokens, blocks, a.w.world) == 64
             ? coop(moe_combine_dot_kernel<64>, a, blocks, 0, stream, 64 * kCombineSubs<64>, kCombineSubs<64>, 1)
             : coop(moe_combine_dot_kernel<256>, a, blocks, 0, stream, 256 * kCombineSubs<256>, kCombineSubs<256>, 2);
}

int launchMoeDequant(const void* q, const float* scales, void* out, const int* n_rows, int max_rows, int hidden, const int* alias,
                     cudaStream_t stream) {
  if (hidden % 128) return static_cast<int>(cudaErrorInvalidValue);
  return static_cast<int>(launchOverlapped(moe_dequant_kernel, dim3(deviceSmCount() * 8), dim3(256), 0, stream, 1, static_cast<const uint8_t*>(q),
                                           scales, static_cast<__nv_bfloat16*>(out), n_rows, max_rows, hidden, alias));
}

int launchMoeExpand(const void* x, const int* ids, const int* dst_rows, const float* probs, void* out, int tokens, int topk, int hidden,
                    cudaStream_t stream) {
  if (tokens <= 0) return 0;
  if (hidden % 128 || topk < 1 || topk > 8) return static_cast<int>(cudaErrorInvalidValue);
  const long long items = static_cast<long long>(tokens) * ((hidden / 8 + 31) / 32);
  return static_cast<int>(launchOverlapped(moe_expand_kernel, dim3(static_cast<unsigned>((items + 7) / 8)), dim3(256), 0, stream, 1,
                                           static_cast<const __nv_bfloat16*>(x), ids, dst_rows, probs, static_cast<__nv_bfloat16*>(out), tokens, topk, hidden));
}

int launchMoeReduceGroups(const void* y, void* z, const int* alias, const void* groups, const int* n_rows, int max_rows, int hidden,
                          cudaStream_t stream) {
  if (hidden % 8 || !alias || !groups) return static_cast<int>(cudaErrorInvalidValue);
  return static_cast<int>(launchOverlapped(moe_reduce_groups_kernel, dim3(deviceSmCount() * 8), dim3(256), 0, stream, 1,
                                           static_cast<const __nv_bfloat16*>(y), static_cast<__nv_bfloat16*>(z), alias,
                                           static_cast<const uint32_t*>(groups), n_rows, max_rows, hidden));
}

int launchQuantFp8Rows(const void* x, void* q, float* scales, long long rows, int hidden, cudaStream_t stream) {
  if (hidden % 128 || rows <= 0) return static_cast<int>(cudaErrorInvalidValue);
  const long long nvec = rows * (hidden >> 3), most = deviceSmCount() * 8ll;       // 256-thread CTAs resident at once
  auto go = [&](auto kern, long long blocks) {
    return static_cast<int>(launchOverlapped(kern, dim3(static_cast<unsigned>(blocks < most ? blocks : most)), dim3(256), 0, stream, 1,
                                             static_cast<const __nv_bfloat16*>(x), static_cast<uint8_t*>(q), scales, nvec));
  };
  return nvec <= most * 256 ? go(quant_rows_kernel<1>, (nvec + 255) / 256) : go(quant_rows_kernel<4>, (nvec + 1023) / 1024);
}

int launchQuantFp8Blocks(const void* w, void* q, float* scales, int rows, int cols, cudaStream_t stream) {
  if (rows % 128 || cols % 128 || rows <= 0 || cols <= 0) return static_cast<int>(cudaErrorInvalidValue);
  dim3 grid(cols / 128, rows / 128);
  quant_blocks_kernel<<<grid, 256, 0, stream>>>(static_cast<const __nv_bfloat16*>(w), static_cast<uint8_t*>(q), scales, rows, cols);
  return static_cast<int>(cudaGetLastError());
}

int launchMoeRoute(const float* logits, int* ids, float* probs, int* pos, int* counts, int tokens, int experts, int topk,
                   cudaStream_t stream) {
  if (experts < 1 || experts > 1024 || topk > experts || tokens <= 0) return static_cast<int>(cudaErrorInvalidValue);
  const int per = (experts + 31) / 32;
  const bool shared = experts <= 256 && tokens * static_cast<long long>(topk) > 8ll * experts;
  auto go = [&](auto kern) {
    int warps = shared ? 32 : 8;
    // few tokens: smaller blocks on more SMs (the 32 warps of a block share the issue slots of one SM)
    while (shared && warps > 2 && (tokens + warps - 1) / warps < deviceSmCount()) warps /= 2;
    return static_cast<int>(launchOverlapped(kern, dim3((tokens + warps - 1) / warps), dim3(32 * warps), shared ? experts * sizeof(int) : 0, stream, 1,
                                             logits, ids, probs, pos, counts, tokens, experts, topk));
  };
  if (per <= 1) return shared ? go(moe_route_kernel<1, true>) : go(moe_route_kernel<1, false>);
  if (per <= 4) return shared ? go(moe_route_kernel<4, true>) : go(moe_route_kernel<4, false>);
  if (per <= 8) return shared ? go(moe_route_kernel<8, true>) : go(moe_route_kernel<8, false>);
  return per <= 16 ? go(moe_route_kernel<16, false>) : go(moe_route_kernel<32, false>);
}

int launchMoeRouteBackward(const float* logits, const int* ids, const float* dprobs, float* dlogits, int tokens, int experts, int topk,
                           cudaStream_t stream) {
  if (experts < 1 || experts > 1024 || topk > experts || tokens <= 0) return static_cast<int>(cudaErrorInvalidValue);
  auto go = [&](auto kern) {
    return static_cast<int>(launchOverlapped(kern, dim3((tokens + 7) / 8), dim3(256), 0, stream, 1, logits, ids, dprobs, dlogits, tokens, experts, topk));
  };
  const int per = (experts + 31) / 32;
  return per <= 1 ? go(moe_route_backward_kernel<1>) : per <= 4 ? go(moe_route_backward_kernel<4>) : per <= 8 ? go(moe_route_backward_kernel<8>)
                                                                                              : go(moe_route_backward_kernel<32>);
}

int launchMoePlan(const int* counts_all, const int* ids, const int* pos, int* rows, int* row_off, int world, int rank, int experts,
                  int tokens, int topk, int cap, cudaStream_t stream) {
  if (experts % world || tokens <= 0) return static_cast<int>(cudaErrorInvalidValue);
  int grid = (tokens * topk + 255) / 256;
  if (grid > 148) grid = 148;
  return static_cast<int>(launchOverlapped(moe_plan_kernel, dim3(grid), dim3(256), (experts + 1) * sizeof(int), stream, 1, counts_all, ids, pos, rows,
                                           row_off, world, rank, experts, tokens, topk, cap));
}

int gemmGroupedBf16(const void* A, int64_t lda, const void* B, int64_t ldb, void* D, int64_t ldd, const int* row_off,
                    int groups, int max_rows, int N, int K, uint32_t flags, void* D2, int sms, uint32_t* status, cudaStream_t stream) {
  if (groups <= 0 || max_rows <= 0) return 0;
  if ((lda | ldb | ldd) % 8) return static_cast<int>(cudaErrorInvalidValue);
  const bool w_mn = flags & GEMM_B_MN;
  if (((flags & (GEMM_GELU | GEMM_DGELU)) && (!D2 || reinterpret_cast<uintptr_t>(D2) % 8)) || (w_mn && K % BK)) return static_cast<int>(cudaErrorInvalidValue);
  CUtensorMap ta, tb;
  std::string err;
  int n_sm = deviceSmCount();
  if (sms > 0 && sms < n_sm) n_sm = sms;
  if (N % 4 == 0 && reinterpret_cast<uintptr_t>(D) % 8 == 0 && n_sm >= 2) {
    // operands exchanged: weights on the M side, the groups' rows on an N side that is cut to the rows there are
    CUtensorMap tw;
    RaggedMaps tx;
    if (!w_mn ? !makeTensorMap2D(&tw, B, TM_BF16, K, static_cast<uint64_t>(groups) * N, ldb, BK, 128, &err)
              : !makeTensorMap2D(&tw, B, TM_BF16, N, static_cast<uint64_t>(groups) * K, ldb, 64, BK, &err))
      return static_cast<int>(cudaErrorInvalidValue);
    for (int i = 0; i < 5; ++i)
      if (!makeTensorMap2D(&tx.x[i], A, TM_BF16, K, max_rows, lda, BK, 128 >> i, &err)) return static_cast<int>(cudaErrorInvalidValue);
    static bool set[2] = {false, false};
    auto go = [&](auto kern, auto epi, bool* done) {
      if (!*done) {
        cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, gemm2::SMEM_BYTES);
        if (e != cudaSuccess) return static_cast<int>(e);
        *done = true;
      }
      return static_cast<int>(launchOverlapped(kern, dim3(n_sm & ~1), dim3(gemm2::NUM_THREADS_WIDE), gemm2::SMEM_BYTES, stream, 2, tw, tx, epi, groups, K, status));
    };
    if (w_mn)
      return go(gemm_grouped_ragged_kernel<true>,
                RaggedEpi<true>{static_cast<__nv_bfloat16*>(D), static_cast<__nv_bfloat16*>(D2), ldd, row_off, N, K, flags, 0}, &set[1]);
    return go(gemm_grouped_ragged_kernel<false>,
              RaggedEpi<false>{static_cast<__nv_bfloat16*>(D), static_cast<__nv_bfloat16*>(D2), ldd, row_off, N, K, flags, 0}, &set[0]);
  }
  if (flags & ~static_cast<uint32_t>(GEMM_GELU_INPLACE)) return static_cast<int>(cudaErrorInvalidValue);
  if (!makeTensorMap2D(&ta, A, TM_BF16, K, max_rows, lda, BK, BM, &err)) return static_cast<int>(cudaErrorInvalidValue);
  if (!makeTensorMap2D(&tb, B, TM_BF16, K, static_cast<uint64_t>(groups) * N, ldb, BK, BN, &err)) return static_cast<int>(cudaErrorInvalidValue);
  GroupedEpi epi{static_cast<__nv_bfloat16*>(D), ldd, row_off, N, flags};
  static bool set = false;
  if (!set) {
    cudaError_t e = cudaFuncSetAttribute(gemm_grouped_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM_BYTES);
    if (e != cudaSuccess) return static_cast<int>(e);
    set = true;
  }
  gemm_grouped_kernel<<<n_sm, NUM_THREADS, SMEM_BYTES, stream>>>(ta, tb, epi, groups, K, status);
  return static_cast<int>(cudaGetLastError());
}

int gemmGroupedWgrad(const GemmProblem& p0, const GemmProblem& p1, const int* row_off, int groups, int max_rows, void* maps, uint32_t* status,
                     cudaStream_t stream) {
  if (groups <= 0) return 0;
  const GemmProblem* ps[2] = {&p0, &p1};
  WgradTemplates tm;
  WgradEpi epi{};
  std::string err;
  long long tiles = 0;
  for (int q = 0; q < 2; ++q) {
    const GemmProblem& p = *ps[q];
    if (max_rows <= 0 || p.M <= 0 || p.N <= 0 || (p.lda | p.ldb | p.ldd) % 8 || p.accumulate ||
        (reinterpret_cast<uintptr_t>(p.A) | reinterpret_cast<uintptr_t>(p.B) | reinterpret_cast<uintptr_t>(p.D)) % 16)
      return static_cast<int>(cudaErrorInvalidValue);
    if (!makeTensorMap2D(&tm.m[2 * q], p.A, TM_BF16, p.M, max_rows, p.lda, 64, gemm2::BK, &err) ||
        !makeTensorMap2D(&tm.m[2 * q + 1], p.B, TM_BF16, p.N, max_rows, p.ldb, 64, gemm2::BK, &err))
      return static_cast<int>(cudaErrorInvalidValue);
    epi.e[q] = StoreEpi{p.D, nullptr, nullptr, p.ldd, p.M, p.N, 0u};
    tiles += static_cast<long long>(groups) * ((p.M + 255) / 256) * ((p.N + 255) / 256);
  }
  if (reinterpret_cast<uintptr_t>(maps) % 128) return static_cast<int>(cudaErrorInvalidValue);
  epi.row_off = row_off;
  epi.maps = static_cast<const CUtensorMap*>(maps);
  static bool set = false;
  if (!set) {
    cudaError_t e = cudaFuncSetAttribute(gemm_grouped_wgrad_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, gemm2::SMEM_BYTES);
    if (e != cudaSuccess) return static_cast<int>(e);
    set = true;
  }
  wgrad_maps_kernel<<<groups, 128, 0, stream>>>(tm, row_off, max_rows, static_cast<CUtensorMap*>(maps));
  const int pairs = deviceSmCount() / 2;
  return static_cast<int>(launchOverlapped(gemm_grouped_wgrad_kernel, dim3(2 * static_cast<int>(tiles < pairs ? tiles : pairs)),
                                           dim3(gemm2::NUM_THREADS_WIDE), gemm2::SMEM_BYTES, stream, 2, epi, groups, status));
}

}  // namespace pccl
