// LayerNorm forward and backward for bf16 activations (fp32 statistics).  Forward: a group of warps per row; every
// thread keeps its 8-element vectors of the row in registers, so x is read once.  Backward: a group of warps
// per row (as many as cover it), several rows at a time, x and dy read once; the kernel is persistent, its
// threads keep their columns' share of dgamma / dbeta in registers across all of their rows, and each CTA writes
// one partial row at the end; a second small kernel adds the partial rows.  (PyTorch's stock backward takes two
// kernels and ~230 us per call at 16384 x 2048.)
//
// Both directions can carry the residual connection that surrounds the norm in a pre-norm transformer block:
// forward takes `delta` and computes s = x + delta (stored, it is the next residual stream) and y = LN(s) in one
// pass; backward adds the gradient that arrives on the residual stream (`dres`) to the norm's input gradient, and
// can emit the column sums of that total -- the bias gradient of the linear layer that produced `delta` -- next
// to dgamma / dbeta.  That removes the separate element-wise add kernels and one pass per bias gradient.
#include <cuda_bf16.h>

#include <initializer_list>

#include "api.h"
#include "elementwise_api.h"
#include "launch.h"
#include "prims.cuh"

namespace pccl {

namespace {

using namespace dev;

// Forward.  A group of `gw` warps owns a row with up to four 16-byte vectors per thread: all loads of a row are out before the first sum, and a
// row of one warp (D <= 1024) takes no barrier.  A row stays in registers as it came, eight values in four registers, and scale and shift
// are read last (they are in L1 or L2).  A CTA is ONE_ROW, or as many rows as its 256 threads hold; the groups' barriers of the latter are named
// at run time, for which a CTA sets all 16 barriers aside, and an SM then holds few of them.  layerNormFwdForm (below) says which runs where.
// Memory bounds it: cold L2, us, plain and with the residual sum, 16384 x 2048 36, 49 (5.5 TB/s); 16384 x 1024 21, 29; 16384 x 256 12, 14;
// 4096 x 8192 33, 50.  With two vectors per thread, CTAs of 128 threads or scale and shift ahead of the sums 16384 x 2048 takes 53, 55 and 51.
template <int VPT, bool ONE_ROW>
__global__ void __launch_bounds__(256, ONE_ROW ? (VPT == 1 ? 8 : VPT == 2 ? 6 : 5) : VPT == 4 ? 4 : 1)
ln_fwd_kernel(const __nv_bfloat16* x, const __nv_bfloat16* delta, __nv_bfloat16* sum_out, const __nv_bfloat16* gamma, const __nv_bfloat16* beta,
              __nv_bfloat16* y, float* mean, float* rstd, long long rows, int D, float eps, int gw) {
  __shared__ float part[2][8];                              // [sum, squares][warp]
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int group = ONE_ROW ? 0 : warp / gw, groups = ONE_ROW ? 1 : (blockDim.x >> 5) / gw, tid = threadIdx.x - group * gw * 32;
  const int nvec = D >> 3, width = gw * 32;
  dev::pdl_launch();
  dev::pdl_wait();
  const long long row = static_cast<long long>(blockIdx.x) * groups + group;
  if (row >= rows) return;                                  // the whole group: barriers are per group
  const long long at = row * D + tid * 8;
  const Vec16 zero{{0u, 0u, 0u, 0u}};
  Vec16 v[VPT];
#pragma unroll
  for (int j = 0; j < VPT; ++j) v[j] = tid + j * width < nvec ? ld16(x + at + j * width * 8) : zero;
  if (delta) {
    Vec16 g[VPT];
#pragma unroll
    for (int j = 0; j < VPT; ++j) g[j] = tid + j * width < nvec ? ld16(delta + at + j * width * 8) : zero;
#pragma unroll
    for (int j = 0; j < VPT; ++j) {
      // the norm sees the sum as it is stored (rounded to bf16), so that backward, which re-reads it, agrees
      float f[8], d[8];
      unpack<DT_BF16>(v[j], f);
      unpack<DT_BF16>(g[j], d);
#pragma unroll
      for (int k = 0; k < 8; ++k) f[k] += d[k];
      v[j] = pack<DT_BF16>(f);
      if (tid + j * width < nvec) st16(sum_out + at + j * width * 8, v[j]);
    }
  }
  auto group_sum = [&](float t, int which) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
    if (!ONE_ROW && gw == 1) return t;
    if (lane == 0) part[which][warp] = t;
    if (ONE_ROW) __syncthreads();
    else asm volatile("bar.sync %0, %1;" ::"r"(group + 1), "r"(width) : "memory");
    t = 0.f;
    for (int w = 0; w < gw; ++w) t += part[which][group * gw + w];
    return t;
  };
  float s = 0.f;
#pragma unroll
  for (int j = 0; j < VPT; ++j) {
    float f[8];
    unpack<DT_BF16>(v[j], f);                               // vectors past the row are zeros
#pragma unroll
    for (int k = 0; k < 8; ++k) s += f[k];
  }
  const float mu = group_sum(s, 0) / D;
  float q = 0.f;
#pragma unroll
  for (int j = 0; j < VPT; ++j) {
    if (tid + j * width < nvec) {
      float f[8];
      unpack<DT_BF16>(v[j], f);
#pragma unroll
      for (int k = 0; k < 8; ++k) { const float d = f[k] - mu; q += d * d; }
    }
  }
  const float rs = rsqrtf(group_sum(q, 1) / D + eps);
  if (tid == 0 && mean) { mean[row] = mu; rstd[row] = rs; }
#pragma unroll
  for (int j = 0; j < VPT; ++j) {
    if (tid + j * width < nvec) {
      const Vec16 g = ld16(gamma + (tid + j * width) * 8), b = ld16(beta + (tid + j * width) * 8);
      float f[8], gf[8], bf[8], o[8];
      unpack<DT_BF16>(v[j], f);
      unpack<DT_BF16>(g, gf);
      unpack<DT_BF16>(b, bf);
#pragma unroll
      for (int k = 0; k < 8; ++k) o[k] = (f[k] - mu) * rs * gf[k] + bf[k];
      st16(y + at + j * width * 8, pack<DT_BF16>(o));
    }
  }
}

// Sums of N values (a power of two) over a group of `gw` warps (those from `first` on); every thread gets them.  The lanes of a warp halve
// the values among them as they add up, so eight values take 9 shuffles where a butterfly each takes 40, and a warp reads each word of
// `stat` ([warp][N]) once where every thread did.  `bar` is the group's barrier.
template <int N>
__device__ __forceinline__ void group_sum(float (&v)[N], float (*stat)[N], int warp, int lane, int gw, int first, int bar) {
  int idx = 0;
#pragma unroll
  for (int n = N / 2, o = 1; n > 0; n /= 2, o *= 2) {
    const bool up = lane & o;
#pragma unroll
    for (int i = 0; i < n; ++i) {
      const float send = up ? v[i] : v[i + n], keep = up ? v[i + n] : v[i];
      v[i] = keep + __shfl_xor_sync(0xffffffffu, send, o);
    }
    idx += up ? n : 0;
  }
  float t = v[0];
#pragma unroll
  for (int o = N; o < 32; o *= 2) t += __shfl_xor_sync(0xffffffffu, t, o);
  if (gw == 1) {
#pragma unroll
    for (int i = 0; i < N; ++i) {
      int from = 0;                                          // the lane below N whose idx is i
#pragma unroll
      for (int n = N / 2, o = 1; n > 0; n /= 2, o *= 2) from += i & n ? o : 0;
      v[i] = __shfl_sync(0xffffffffu, t, from);
    }
    return;
  }
  if (lane < N) stat[warp][idx] = t;
  asm volatile("bar.sync %0, %1;" ::"r"(bar), "r"(gw * 32) : "memory");
  t = 0.f;
  for (int w = lane / N; w < gw; w += 32 / N) t += stat[first + w][lane & (N - 1)];
#pragma unroll
  for (int o = N; o < 32; o *= 2) t += __shfl_xor_sync(0xffffffffu, t, o);
#pragma unroll
  for (int i = 0; i < N; ++i) v[i] = __shfl_sync(0xffffffffu, t, i);
}

// Two fp32 values in one 64-bit register pair: one instruction adds or multiplies both.
__device__ __forceinline__ uint64_t pair(float a, float b) {
  uint64_t r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
  return r;
}
__device__ __forceinline__ float2 split(uint64_t p) {
  float2 r;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(p));
  return r;
}
__device__ __forceinline__ uint64_t add2(uint64_t a, uint64_t b) {
  uint64_t r;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ uint64_t mul2(uint64_t a, uint64_t b) {
  uint64_t r;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ uint64_t fma2(uint64_t a, uint64_t b, uint64_t c) {
  uint64_t r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
  return r;
}
__device__ __forceinline__ uint64_t pair_of(uint32_t bf16x2) {
  return pair(__uint_as_float(bf16x2 << 16), __uint_as_float(bf16x2 & 0xffff0000u));
}
__device__ __forceinline__ uint32_t bf16x2_of(uint64_t p) {
  const float2 f = split(p);
  uint32_t r;
  asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(r) : "f"(f.y), "f"(f.x));
  return r;
}

// 16 bytes to shared memory behind the thread's back; only the first `n` of them are read, the rest become zeros.
__device__ __forceinline__ void cp_async16(void* dst, const void* src, int n) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(static_cast<uint32_t>(__cvta_generic_to_shared(dst))), "l"(src), "r"(n) : "memory");
}

// Backward.  A group of `gw` warps owns a row -- as many as cover it with VPT 16-byte vectors per thread (one up to D = 2048) -- and takes
// R rows at a time: R x VPT x 3 vectors are in flight per thread, and the row statistics of all R rows cross the group in one exchange.
// The next R rows are fetched into registers while these are worked on (STAGES = 0), as far as that goes without spills, which cost
// far more than the fetch brings.  Beyond D = 2048 many rows of the EXTRA form come through a ring in shared memory, STAGES - 1 trips ahead.
// A thread copies only what it reads itself, so no barrier guards the ring, and a slot is filled again one trip after its values were
// used.  (Where the registers hold the next rows a ring brings nothing: 16384 x 2048 52 with either.)  Few rows gain nothing from a ring and
// pay for its filling: they come straight into registers, beyond D = 4096 each trip's own (STAGES = -1: no registers for the next).
// us, ring / without: 1 x 3072 5.7 / 4.6, 600 x 4096 12.4 / 11.3, 1531 x 4096 17.2 / 15.5, 2331 x 3072 16.4 / 15.8, 3000 x 2560 18.4 / 19.4; 1 x 8192
// 9.9 / 9.1, 600 x 5120 14.8 / 13.6, 1000 x 6144 18.9 / 17.8, 1531 x 5120 23.0 / 23.9, 4096 x 8192 60 / 79.
// A thread keeps the same columns for all of its rows, so the column sums (dgamma, dbeta, bias gradient) stay in registers; the CTA's
// groups add theirs up at the end and write one partial row per array.
// With eight warps per SM the instructions count beside the memory: the arithmetic is on pairs (f32x2) and the exchange is group_sum.
// Times, us, 20 calls in a row (a butterfly per sum, one value per instruction, no ring -> now): EXTRA 16384 x 2048 57.7 -> 51.7 (5.2 TB/s),
// 16384 x 1536 57.3 -> 46.0, 16384 x 512 18.9 -> 15.4, 2331 x 768 9.5 -> 8.6, 20000 x 2560 115 -> 90, 8192 x 4096 57.7 -> 55.1, 4096 x 8192
// 74.3 -> 60.4, 256 x 8192 15.2 -> 16.1; plain 16384 x 2048 46.6 -> 44.1, 16384 x 1536 40.2 -> 37.7, 8192 x 4096 44.7 -> 43.9.
template <int VPT, int R, bool EXTRA, int CTAS, int STAGES, int THREADS>
__global__ void __launch_bounds__(THREADS, CTAS) ln_bwd_kernel(const __nv_bfloat16* dy, const __nv_bfloat16* x, const __nv_bfloat16* gamma,
                                                           const float* mean, const float* rstd, const __nv_bfloat16* dres, __nv_bfloat16* dx,
                                                           float* part_g, float* part_b, float* part_c, long long rows, int D, int gw) {
  __shared__ float stat[2][THREADS / 32][2 * R];                       // [parity][warp][value]: partial sums of a warp
  extern __shared__ __align__(16) float group_sums[];       // [groups][arrays][D], with more than one group
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int group = warp / gw, groups = (blockDim.x >> 5) / gw, tid = threadIdx.x - group * gw * 32;
  const int nvec = D >> 3, width = gw * 32;
  dev::pdl_launch();
  dev::pdl_wait();
  const Vec16 zero{{0u, 0u, 0u, 0u}};
  Vec16 g[VPT];
  uint64_t ag[VPT][4], ab[VPT][4], ac[EXTRA ? VPT : 1][4];
#pragma unroll
  for (int j = 0; j < VPT; ++j) {
    g[j] = tid + j * width < nvec ? ld16(gamma + (tid + j * width) * 8) : zero;
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      ag[j][k] = 0;
      ab[j][k] = 0;
      if (EXTRA) ac[EXTRA ? j : 0][k] = 0;
    }
  }
  const float inv_d = 1.0f / D;
  const long long step = static_cast<long long>(gridDim.x) * groups * R;
  struct Rows {
    Vec16 x[R][VPT], d[R][VPT], r[EXTRA ? R : 1][VPT];
    float mu[R], rs[R];
  };
  auto load = [&](Rows& t, long long row0) {
#pragma unroll
    for (int r = 0; r < R; ++r) {
      const long long at = (row0 + r) * D + tid * 8;
#pragma unroll
      for (int j = 0; j < VPT; ++j) {
        const bool in = row0 + r < rows && tid + j * width < nvec;
        t.x[r][j] = in ? ld16(x + at + j * width * 8) : zero;
        t.d[r][j] = in ? ld16(dy + at + j * width * 8) : zero;
        if (EXTRA) t.r[EXTRA ? r : 0][j] = in && dres ? ld16(dres + at + j * width * 8) : zero;
      }
      t.mu[r] = row0 + r < rows ? mean[row0 + r] : 0.f;
      t.rs[r] = row0 + r < rows ? rstd[row0 + r] : 0.f;
    }
  };
  long long row0 = (static_cast<long long>(blockIdx.x) * groups + group) * R;
  Rows cur;
  constexpr int ARR = EXTRA ? 3 : 2, SLOTS = STAGES > 0 ? STAGES : 1;
  Vec16* ring = reinterpret_cast<Vec16*>(group_sums);       // [STAGES][R][ARR][VPT][THREADS]
  auto slot_of = [&](int slot, int r, int a, int j) { return ring + (((slot * R + r) * ARR + a) * VPT + j) * THREADS + threadIdx.x; };
  auto fetch = [&](int slot, long long row0) {
#pragma unroll
    for (int r = 0; r < R; ++r) {
#pragma unroll
      for (int j = 0; j < VPT; ++j) {
        const bool in = row0 + r < rows && tid + j * width < nvec;
        const long long at = in ? (row0 + r) * D + (tid + j * width) * 8 : 0;
        const int n = in ? 16 : 0;                          // nothing is read where this is 0, the slot becomes zeros
        cp_async16(slot_of(slot, r, 0, j), x + at, n);
        cp_async16(slot_of(slot, r, 1, j), dy + at, n);
        if (EXTRA) cp_async16(slot_of(slot, r, ARR - 1, j), dres ? dres + at : x, dres ? n : 0);
      }
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  float mu_next[R], rs_next[R];
  auto stats = [&](long long row0) {
#pragma unroll
    for (int r = 0; r < R; ++r) {
      mu_next[r] = row0 + r < rows ? mean[row0 + r] : 0.f;
      rs_next[r] = row0 + r < rows ? rstd[row0 + r] : 0.f;
    }
  };
  if (STAGES > 0) {
#pragma unroll
    for (int i = 0; i < STAGES - 1; ++i) fetch(i, row0 + i * step);
    stats(row0);
  } else if (STAGES == 0) {
    load(cur, row0);
  }
  int parity = 0, slot = 0;
  for (; row0 < rows; row0 += step, parity ^= 1, slot = slot + 1 == SLOTS ? 0 : slot + 1) {
    if (STAGES < 0) load(cur, row0);
    if (STAGES > 0) {
      asm volatile("cp.async.wait_group %0;" ::"n"(STAGES > 1 ? STAGES - 2 : 0) : "memory");
#pragma unroll
      for (int r = 0; r < R; ++r) {
        cur.mu[r] = mu_next[r];
        cur.rs[r] = rs_next[r];
#pragma unroll
        for (int j = 0; j < VPT; ++j) {
          cur.x[r][j] = *slot_of(slot, r, 0, j);
          cur.d[r][j] = *slot_of(slot, r, 1, j);
          if (EXTRA) cur.r[EXTRA ? r : 0][j] = *slot_of(slot, r, ARR - 1, j);
        }
      }
      fetch(slot == 0 ? SLOTS - 1 : slot - 1, row0 + (STAGES - 1) * step);     // the slot of the trip before
      stats(row0 + step);
    }
    float sums[2 * R];                     // per row: of dy * gamma, and of that times the normalised x
#pragma unroll
    for (int r = 0; r < R; ++r) {
      uint64_t s1 = 0, s2 = 0;
      const uint64_t nmu = pair(-cur.mu[r], -cur.mu[r]), rs = pair(cur.rs[r], cur.rs[r]);
#pragma unroll
      for (int j = 0; j < VPT; ++j) {
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          const uint64_t dg = mul2(pair_of(cur.d[r][j].w[k]), pair_of(g[j].w[k])), xh = mul2(add2(pair_of(cur.x[r][j].w[k]), nmu), rs);
          s1 = add2(s1, dg);
          s2 = fma2(dg, xh, s2);
        }
      }
      sums[2 * r] = split(s1).x + split(s1).y;
      sums[2 * r + 1] = split(s2).x + split(s2).y;
    }
    Rows next;
    if (STAGES == 0) load(next, row0 + step);  // on its way behind the exchange, the arithmetic and the stores
    // the other parity's slots are not written again before every warp of the group has passed this barrier once more
    group_sum<2 * R>(sums, stat[parity], warp, lane, gw, group * gw, group + 1);
#pragma unroll
    for (int r = 0; r < R; ++r) {
      const float m1 = sums[2 * r] * inv_d, m2 = sums[2 * r + 1] * inv_d;
      const uint64_t nm1 = pair(-m1, -m1), nm2 = pair(-m2, -m2), nmu = pair(-cur.mu[r], -cur.mu[r]), rs = pair(cur.rs[r], cur.rs[r]);
#pragma unroll
      for (int j = 0; j < VPT; ++j) {
        Vec16 out;
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          const uint64_t d = pair_of(cur.d[r][j].w[k]), xh = mul2(add2(pair_of(cur.x[r][j].w[k]), nmu), rs);
          uint64_t o = fma2(xh, nm2, fma2(d, pair_of(g[j].w[k]), nm1));
          if (EXTRA) {
            o = fma2(o, rs, pair_of(cur.r[EXTRA ? r : 0][j].w[k]));
            ac[EXTRA ? j : 0][k] = add2(ac[EXTRA ? j : 0][k], o);
          } else {
            o = mul2(o, rs);
          }
          ag[j][k] = fma2(d, xh, ag[j][k]);
          ab[j][k] = add2(ab[j][k], d);
          out.w[k] = bf16x2_of(o);
        }
        if (row0 + r < rows && tid + j * width < nvec) st16(dx + (row0 + r) * D + (tid + j * width) * 8, out);
      }
    }
    if (STAGES == 0) cur = next;
  }
  if (STAGES > 0) {
    asm volatile("cp.async.wait_all;" ::: "memory");        // the last trips fetched zeros
    __syncthreads();
  }
  const int arrays = EXTRA && part_c ? 3 : 2;
#pragma unroll
  for (int j = 0; j < VPT; ++j) {
    const int v = tid + j * width;
    if (v >= nvec) continue;
#pragma unroll
    for (int a = 0; a < (EXTRA ? 3 : 2); ++a) {
      if (a >= arrays) continue;
      const uint64_t* f = a == 0 ? ag[j] : a == 1 ? ab[j] : ac[EXTRA ? j : 0];
      float* dst = groups > 1 ? group_sums + (group * 3 + a) * D + v * 8
                              : (a == 0 ? part_g : a == 1 ? part_b : part_c) + static_cast<long long>(blockIdx.x) * D + v * 8;
      *reinterpret_cast<float4*>(dst) = make_float4(split(f[0]).x, split(f[0]).y, split(f[1]).x, split(f[1]).y);
      *reinterpret_cast<float4*>(dst + 4) = make_float4(split(f[2]).x, split(f[2]).y, split(f[3]).x, split(f[3]).y);
    }
  }
  if (groups > 1) {
    __syncthreads();
    for (int i = threadIdx.x; i < arrays * D; i += blockDim.x) {
      const int a = i / D, c = i - a * D;
      float t = 0.f;
      for (int q = 0; q < groups; ++q) t += group_sums[(q * 3 + a) * D + c];
      (a == 0 ? part_g : a == 1 ? part_b : part_c)[static_cast<long long>(blockIdx.x) * D + c] = t;
    }
  }
}

// Adds the partial rows of up to three arrays [nparts, D] column by column into bf16 vectors of length D.  A CTA owns
// 32 columns of one array (blockIdx.y); its 32 warps each walk every 32nd partial row, so the rows are read 32 at a time with
// full coalescing.
struct ReduceJob {
  const float* part[3];
  __nv_bfloat16* out[3];
  float* add;              // fp32 vector that grows by the sums of the first array instead of out[0], or null
};

__global__ void __launch_bounds__(1024) partial_rows_reduce_kernel(ReduceJob job, int nparts, int D) {
  __shared__ float sm[32][33];
  dev::pdl_launch();
  dev::pdl_wait();
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int col = blockIdx.x * 32 + lane;
  const float* part = blockIdx.y == 0 ? job.part[0] : blockIdx.y == 1 ? job.part[1] : job.part[2];
  float acc = 0.f;
  if (col < D) {
#pragma unroll 4
    for (int p = warp; p < nparts; p += 32) acc += part[static_cast<long long>(p) * D + col];
  }
  sm[warp][lane] = acc;
  __syncthreads();
  if (warp == 0 && col < D) {
    float t = 0.f;
#pragma unroll
    for (int k = 0; k < 32; ++k) t += sm[k][lane];
    if (job.add) job.add[col] += t;
    else (blockIdx.y == 0 ? job.out[0] : blockIdx.y == 1 ? job.out[1] : job.out[2])[col] = __float2bfloat16_rn(t);
  }
}

// Column sums of a bf16 matrix [rows, N] (row stride ld): the bias gradient of a linear layer whose output gradient
// comes from elsewhere.  A CTA owns 256 columns (one 16-byte vector per lane, 8 warps = 8 rows at a time) and a block
// of rows; it writes one partial row, which partial_rows_reduce_kernel adds up.
__global__ void __launch_bounds__(256) colsum_partial_kernel(const __nv_bfloat16* x, long long ld, long long rows, int N,
                                                             int rows_per_part, float* part) {
  __shared__ float sm[8][256 + 8];
  dev::pdl_launch();
  dev::pdl_wait();
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int col = blockIdx.x * 256 + lane * 8;
  const long long r0 = static_cast<long long>(blockIdx.y) * rows_per_part;
  const long long r1 = r0 + rows_per_part < rows ? r0 + rows_per_part : rows;
  float acc[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
  if (col < N) {
    long long r = r0 + warp;
    for (; r + 56 < r1; r += 64) {         // eight independent loads in flight
      Vec16 v[8];
#pragma unroll
      for (int i = 0; i < 8; ++i) v[i] = ld16(x + (r + 8 * i) * ld + col);
#pragma unroll
      for (int i = 0; i < 8; i += 2) {
        float a[8], b[8];
        unpack<DT_BF16>(v[i], a);
        unpack<DT_BF16>(v[i + 1], b);
#pragma unroll
        for (int k = 0; k < 8; ++k) acc[k] += a[k] + b[k];
      }
    }
    for (; r < r1; r += 8) {
      float a[8];
      unpack<DT_BF16>(ld16(x + r * ld + col), a);
#pragma unroll
      for (int k = 0; k < 8; ++k) acc[k] += a[k];
    }
  }
#pragma unroll
  for (int k = 0; k < 8; ++k) sm[warp][lane * 8 + k] = acc[k];
  __syncthreads();
  const int c = blockIdx.x * 256 + threadIdx.x;
  if (c < N) {
    float t = 0.f;
#pragma unroll
    for (int w = 0; w < 8; ++w) t += sm[w][threadIdx.x];
    part[static_cast<long long>(blockIdx.y) * N + c] = t;
  }
}

// The gradients of q, k and v, each [batch, heads, seq, hd] with the given strides, become the gradient of the packed
// projection output [batch * seq, 3, heads, hd] in one pass that also sums its columns (the projection's bias gradient): a copy
// and a column-sum kernel otherwise read the 3 x rows x width values once more.  A CTA owns 256 output columns (one vector of
// eight per lane, hd % 8 == 0, so a vector lies in one head of one of the three) and a block of rows, eight at a time.
struct QkvGrads {
  const __nv_bfloat16* g[3];
  long long sb[3], sh[3], st[3];           // strides in elements: batch, head, position
};

__global__ void __launch_bounds__(256) qkv_pack_kernel(QkvGrads in, __nv_bfloat16* out, long long rows, int seq, int heads, int hd,
                                                       int rows_per_part, float* part) {
  __shared__ float sm[8][256 + 8];
  dev::pdl_launch();
  dev::pdl_wait();
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int width = heads * hd, N = 3 * width;
  const int col = blockIdx.x * 256 + lane * 8;
  const long long r0 = static_cast<long long>(blockIdx.y) * rows_per_part;
  const long long r1 = r0 + rows_per_part < rows ? r0 + rows_per_part : rows;
  float acc[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
  if (col < N) {
    const int which = col / width, h = (col - which * width) / hd, d = col - which * width - h * hd;
    const __nv_bfloat16* g = (which == 0 ? in.g[0] : which == 1 ? in.g[1] : in.g[2]) + (which == 0 ? in.sh[0] : which == 1 ? in.sh[1] : in.sh[2]) * h + d;
    const long long sb = which == 0 ? in.sb[0] : which == 1 ? in.sb[1] : in.sb[2], st = which == 0 ? in.st[0] : which == 1 ? in.st[1] : in.st[2];
    for (long long r = r0 + warp; r < r1; r += 64) {
      Vec16 v[8];
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        const long long row = r + 8 * i;
        const long long b = row / seq;
        if (row < r1) v[i] = ld16(g + b * sb + (row - b * seq) * st);
      }
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        const long long row = r + 8 * i;
        if (row >= r1) break;
        st16(out + row * N + col, v[i]);
        float f[8];
        unpack<DT_BF16>(v[i], f);
#pragma unroll
        for (int k = 0; k < 8; ++k) acc[k] += f[k];
      }
    }
  }
#pragma unroll
  for (int k = 0; k < 8; ++k) sm[warp][lane * 8 + k] = acc[k];
  __syncthreads();
  const int c = blockIdx.x * 256 + threadIdx.x;
  if (c < N) {
    float t = 0.f;
#pragma unroll
    for (int w = 0; w < 8; ++w) t += sm[w][threadIdx.x];
    part[static_cast<long long>(blockIdx.y) * N + c] = t;
  }
}

// The kernels read and write 16 bytes at a time.
bool aligned16(std::initializer_list<const void*> pointers) {
  uintptr_t bits = 0;
  for (const void* p : pointers) bits |= reinterpret_cast<uintptr_t>(p);
  return bits % 16 == 0;
}

}  // namespace

LayerNormFwdForm layerNormFwdForm(long long rows, int D, int sms) {
  const int nvec = D / 8;
  const long long values = rows * D, mi = 1ll << 20;
  LayerNormFwdForm f{(nvec + 127) / 128, 4, 1, false};
  if (f.warps == 1) f.vectors = (nvec + 31) / 32;
  const bool short_chain = D <= 2048 ? values <= 4 * mi : values <= 7 * mi || D > 5120;
  if (short_chain) {
    f.vectors = (nvec + 255) / 256;
    f.warps = (nvec + 32 * f.vectors - 1) / (32 * f.vectors);
  }
  if (f.warps > 1 && (D > 2048 || short_chain)) f.one_row = rows <= sms || (D > 1024 && rows > 3 * sms);
  if (f.one_row && f.vectors == 2 && f.warps == 8 && rows > 6 * sms && rows <= 8 * sms) f.one_row = false;
  if (!f.one_row && D > 2048) {
    f.vectors = 4;
    f.warps = (nvec + 127) / 128;
  }
  if (f.one_row && f.vectors == 1 && D > 1024 && rows <= 8 * sms) f.warps = 8;
  if (f.one_row) return f;
  f.rows = 8 / f.warps;
  while (f.rows > 1 && (rows + f.rows - 1) / f.rows < sms) f.rows /= 2;
  return f;
}

int launchLayerNormFwd(const void* x, const void* delta, void* sum_out, const void* gamma, const void* beta, void* y, float* mean,
                       float* rstd, long long rows, int D, float eps, cudaStream_t stream) {
  if (rows <= 0) return 0;
  if (D % 8 || D > 8192 || (delta && !sum_out) || !aligned16({x, delta, sum_out, gamma, beta, y})) return static_cast<int>(cudaErrorInvalidValue);
  auto X = static_cast<const __nv_bfloat16*>(x); auto G = static_cast<const __nv_bfloat16*>(gamma);
  auto B = static_cast<const __nv_bfloat16*>(beta); auto Y = static_cast<__nv_bfloat16*>(y);
  auto DL = static_cast<const __nv_bfloat16*>(delta); auto S = static_cast<__nv_bfloat16*>(sum_out);
  const LayerNormFwdForm form = layerNormFwdForm(rows, D, deviceSmCount());
  const unsigned grid = static_cast<unsigned>((rows + form.rows - 1) / form.rows);
  auto go = [&](auto kern) {
    return static_cast<int>(launchOverlapped(kern, dim3(grid), dim3(form.rows * form.warps * 32), 0, stream, 1, X, DL, S, G, B, Y, mean, rstd, rows, D, eps,
                                             form.warps));
  };
  if (form.one_row) {
    return form.vectors == 1 ? go(ln_fwd_kernel<1, true>) : form.vectors == 2 ? go(ln_fwd_kernel<2, true>)
         : form.vectors == 3 ? go(ln_fwd_kernel<3, true>) : go(ln_fwd_kernel<4, true>);
  }
  return form.vectors == 1 ? go(ln_fwd_kernel<1, false>) : form.vectors == 2 ? go(ln_fwd_kernel<2, false>)
       : form.vectors == 3 ? go(ln_fwd_kernel<3, false>) : go(ln_fwd_kernel<4, false>);
}

bool layerNormBwdRing(long long rows, int D, int sms) { return D > 2048 && rows > (D <= 4096 ? 16 : 7) * sms; }

int layerNormBwdParts(long long rows) { return static_cast<int>(rows < 148 * 2 ? rows : 148 * 2); }

int launchLayerNormBwd(const void* dy, const void* x, const void* gamma, const float* mean, const float* rstd, const void* dres, void* dx,
                       void* dgamma, void* dbeta, void* dcolsum, float* partials, long long rows, int D, cudaStream_t stream) {
  if (rows <= 0) return 0;
  if (D % 8 || D > 8192 || !aligned16({dy, x, gamma, dres, dx})) return static_cast<int>(cudaErrorInvalidValue);
  const int most = layerNormBwdParts(rows);
  float* pg = partials;
  float* pb = partials + static_cast<long long>(most) * D;
  float* pc = dcolsum ? partials + 2ll * most * D : nullptr;
  int nparts = 0;
  // VPT vectors per thread, R rows per trip, `sms` CTAs resident per SM, a ring of `slots` bytes
  auto go = [&](auto kern, int vpt, int r, int sms, int threads, size_t slots) {
    const int gw = (D / 8 + 32 * vpt - 1) / (32 * vpt), groups = threads / 32 / gw;
    const long long want = (rows + static_cast<long long>(groups) * r - 1) / (static_cast<long long>(groups) * r);
    const int limit = deviceSmCount() * sms < most ? deviceSmCount() * sms : most;
    nparts = static_cast<int>(want < limit ? want : limit);
    const size_t sums = groups > 1 ? static_cast<size_t>(groups) * 3 * D * sizeof(float) : 0;         // at most 24 KiB per 256 threads
    if (slots) {
      const cudaError_t set = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(slots));
      if (set != cudaSuccess) return static_cast<int>(set);
    }
    return static_cast<int>(launchOverlapped(kern, dim3(nparts), dim3(groups * gw * 32), slots > sums ? slots : sums, stream, 1,
                                             static_cast<const __nv_bfloat16*>(dy), static_cast<const __nv_bfloat16*>(x),
                                             static_cast<const __nv_bfloat16*>(gamma), mean, rstd, static_cast<const __nv_bfloat16*>(dres),
                                             static_cast<__nv_bfloat16*>(dx), pg, pb, pc, rows, D, gw));
  };
  constexpr size_t kRing = 192 * 1024;    // four stages of two rows of up to 4096 values and three arrays, or of one row of up to 8192
  const bool ring = layerNormBwdRing(rows, D, deviceSmCount());
  int e;
  if (!dres && !dcolsum)
    e = D <= 2048 ? go(ln_bwd_kernel<1, 2, false, 2, 0, 256>, 1, 2, 2, 256, 0) : D <= 4096 ? go(ln_bwd_kernel<2, 2, false, 1, 0, 256>, 2, 2, 1, 256, 0)
                                                                                         : go(ln_bwd_kernel<4, 1, false, 1, 0, 256>, 4, 1, 1, 256, 0);
  else if (D <= 2048)
    e = go(ln_bwd_kernel<1, 4, true, 1, 0, 256>, 1, 4, 1, 256, 0);
  else if (D <= 4096)
    e = ring ? go(ln_bwd_kernel<1, 2, true, 1, 4, 512>, 1, 2, 1, 512, kRing) : go(ln_bwd_kernel<2, 2, true, 1, 0, 256>, 2, 2, 1, 256, 0);
  else
    e = ring ? go(ln_bwd_kernel<4, 1, true, 1, 4, 256>, 4, 1, 1, 256, kRing) : go(ln_bwd_kernel<4, 1, true, 1, -1, 256>, 4, 1, 1, 256, 0);
  if (e != 0) return e;
  ReduceJob job{{pg, pb, pc}, {static_cast<__nv_bfloat16*>(dgamma), static_cast<__nv_bfloat16*>(dbeta), static_cast<__nv_bfloat16*>(dcolsum)}, nullptr};
  return static_cast<int>(launchOverlapped(partial_rows_reduce_kernel, dim3((D + 31) / 32, dcolsum ? 3 : 2), dim3(1024), 0, stream, 1, job, nparts, D));
}

int colSumParts(long long rows) { return static_cast<int>((rows + 255) / 256 < 64 ? (rows + 255) / 256 : 64); }

// Row blocks of a column-sum launch: about four CTAs per SM in one go.  With 64 row blocks whatever the width, 16384 x 6144 had 1536
// CTAs for 1184 places and took 54 us; now 50 (201 MB).
static int colSumGrid(long long rows, int N) {
  const int cols = (N + 255) / 256, fit = deviceSmCount() * 4 / cols, parts = colSumParts(rows);
  return fit < 1 ? 1 : parts > fit ? fit : parts;
}

int launchColSum(const void* x, long long ld, long long rows, int N, void* out_bf16, float* partials, cudaStream_t stream) {
  if (rows <= 0 || N <= 0) return 0;
  if (N % 8 || ld % 8 || reinterpret_cast<uintptr_t>(x) % 16) return static_cast<int>(cudaErrorInvalidValue);
  const int cols = (N + 255) / 256, parts = colSumGrid(rows, N);
  const int rows_per_part = static_cast<int>((rows + parts - 1) / parts);
  const int e = static_cast<int>(launchOverlapped(colsum_partial_kernel, dim3(cols, parts), dim3(256), 0, stream, 1,
                                                  static_cast<const __nv_bfloat16*>(x), ld, rows, N, rows_per_part, partials));
  if (e != 0) return e;
  ReduceJob job{{partials, nullptr, nullptr}, {static_cast<__nv_bfloat16*>(out_bf16), nullptr, nullptr}, nullptr};
  return static_cast<int>(launchOverlapped(partial_rows_reduce_kernel, dim3((N + 31) / 32, 1), dim3(1024), 0, stream, 1, job, parts, N));
}

int launchColSumParts(const ColSum& c, int M, int N, cudaStream_t stream) {
  if (!c.out) return 0;
  ReduceJob job{{c.parts, nullptr, nullptr}, {c.f32 ? nullptr : static_cast<__nv_bfloat16*>(c.out), nullptr, nullptr},
                c.f32 ? static_cast<float*>(c.out) : nullptr};
  return static_cast<int>(launchOverlapped(partial_rows_reduce_kernel, dim3((N + 31) / 32, 1), dim3(1024), 0, stream, 1, job, (M + 31) / 32, N));
}

int launchQkvPack(const void* const* grads, const long long* strides, void* out, int batch, int seq, int heads, int hd, void* colsum_bf16,
                  float* partials, cudaStream_t stream) {
  const long long rows = static_cast<long long>(batch) * seq;
  if (rows <= 0) return 0;
  QkvGrads in;
  for (int i = 0; i < 3; ++i) {
    in.g[i] = static_cast<const __nv_bfloat16*>(grads[i]);
    in.sb[i] = strides[3 * i];
    in.sh[i] = strides[3 * i + 1];
    in.st[i] = strides[3 * i + 2];
    if ((in.sb[i] | in.sh[i] | in.st[i]) % 8 || reinterpret_cast<uintptr_t>(grads[i]) % 16) return static_cast<int>(cudaErrorInvalidValue);
  }
  if (hd % 8 || reinterpret_cast<uintptr_t>(out) % 16) return static_cast<int>(cudaErrorInvalidValue);
  const int N = 3 * heads * hd, parts = colSumGrid(rows, N);
  const int rows_per_part = static_cast<int>((rows + parts - 1) / parts);
  const int e = static_cast<int>(launchOverlapped(qkv_pack_kernel, dim3((N + 255) / 256, parts), dim3(256), 0, stream, 1, in,
                                                  static_cast<__nv_bfloat16*>(out), rows, seq, heads, hd, rows_per_part, partials));
  if (e != 0) return e;
  ReduceJob job{{partials, nullptr, nullptr}, {static_cast<__nv_bfloat16*>(colsum_bf16), nullptr, nullptr}, nullptr};
  return static_cast<int>(launchOverlapped(partial_rows_reduce_kernel, dim3((N + 31) / 32, 1), dim3(1024), 0, stream, 1, job, parts, N));
}

}  // namespace pccl
