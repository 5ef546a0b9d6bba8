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

// Forward.  A group of `gw` warps owns a row with up to four 16-byte vectors per thread (one warp up to D = 1024) and a CTA takes as
// many rows as its 256 threads hold: all loads of a row are out before the first sum, and a row of one warp takes no barrier.  A row
// stays in registers as it came, eight values in four registers, and scale and shift are read last (they are in L1 or L2), so that four
// CTAs fit an SM; with two vectors per thread and six CTAs, with CTAs of 128 threads or with scale and shift ahead of the sums 16384 x 2048
// takes 53, 55 and 51 us.
// Memory bounds it.  Times, us, cold L2, plain and with the residual sum (a CTA of 256 threads per row before -> now): 16384 x 2048
// 39 -> 36, 55 -> 49 (5.5 TB/s); 16384 x 1536 37 -> 32, 49 -> 40; 16384 x 1024 33 -> 21, 43 -> 29; 16384 x 256 29 -> 12, 35 -> 14;
// 4096 x 1024 14 -> 11, 16 -> 12; 4096 x 8192 41 -> 37, 64 -> 49; 1531 x 2048 unchanged at 10 and 12.
template <int VPT>
__global__ void __launch_bounds__(256, VPT == 4 ? 4 : 1) ln_fwd_kernel(const __nv_bfloat16* x, const __nv_bfloat16* delta, __nv_bfloat16* sum_out,
                                                     const __nv_bfloat16* gamma, const __nv_bfloat16* beta, __nv_bfloat16* y,
                                                     float* mean, float* rstd, long long rows, int D, float eps, int gw) {
  __shared__ float part[2][8];                              // [sum, squares][warp]
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int group = warp / gw, groups = (blockDim.x >> 5) / gw, tid = threadIdx.x - group * gw * 32;
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
    if (gw == 1) return t;
    if (lane == 0) part[which][warp] = t;
    asm volatile("bar.sync %0, %1;" ::"r"(group + 1), "r"(width) : "memory");
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

// Backward.  A group of `gw` warps owns a row -- as many as cover it with one 16-byte vector per thread and trip (VPT trips; one
// up to D = 2048) -- and takes R rows at a time: R x VPT x 3 vectors are in flight per thread, and the row statistics of all R
// rows cross the group in one exchange.  The next R rows are fetched (AHEAD) while these are worked on, as far as that goes without
// spills, which cost far more than the fetch brings: two vectors per row in the plain form, three and the column sums of dx in the
// EXTRA one.  A thread keeps the same columns for all of its rows, so the column sums (dgamma,
// dbeta, bias gradient) stay in registers; the CTA's groups add theirs up at the end and write one partial row per array.
// Times, us, cold L2 (one warp per row with its sums in shared memory for D = 256, 512, 1024 and 2048, a CTA per row for the rest
// -> now; in brackets three rows on two CTAs per SM without the fetch ahead): EXTRA 16384 x 2048
// 77 -> 64 [77], 16384 x 1024 44 -> 39 [48], 16384 x 256 28 -> 17 [20], 2331 x 768 32 -> 15 [17], 8192 x 4096 136 -> 64 [83], 4096 x 8192
// 220 -> 83; plain 16384 x 2048 64 -> 52 [73] (3.9 TB/s), 16384 x 1024 40 -> 32 [44], 8192 x 4096 101 -> 52 [79], 4096 x 8192 153 -> 56 [81].
template <int VPT, int R, bool EXTRA, bool AHEAD, int CTAS>
__global__ void __launch_bounds__(256, CTAS) ln_bwd_kernel(const __nv_bfloat16* dy, const __nv_bfloat16* x, const __nv_bfloat16* gamma,
                                                           const float* mean, const float* rstd, const __nv_bfloat16* dres, __nv_bfloat16* dx,
                                                           float* part_g, float* part_b, float* part_c, long long rows, int D, int gw) {
  __shared__ float2 stat[2][8][R];                          // [parity][warp][row]: partial sums of a warp
  extern __shared__ __align__(16) float group_sums[];       // [groups][arrays][D], with more than one group
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int group = warp / gw, groups = (blockDim.x >> 5) / gw, tid = threadIdx.x - group * gw * 32;
  const int nvec = D >> 3, width = gw * 32;
  dev::pdl_launch();
  dev::pdl_wait();
  const Vec16 zero{{0u, 0u, 0u, 0u}};
  Vec16 g[VPT];
  float ag[VPT][8], ab[VPT][8], ac[EXTRA ? VPT : 1][8];
#pragma unroll
  for (int j = 0; j < VPT; ++j) {
    g[j] = tid + j * width < nvec ? ld16(gamma + (tid + j * width) * 8) : zero;
#pragma unroll
    for (int k = 0; k < 8; ++k) {
      ag[j][k] = 0.f;
      ab[j][k] = 0.f;
      if (EXTRA) ac[EXTRA ? j : 0][k] = 0.f;
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
  if (AHEAD) load(cur, row0);
  int parity = 0;
  for (; row0 < rows; row0 += step, parity ^= 1) {
    if (!AHEAD) load(cur, row0);
    float s1[R], s2[R];
#pragma unroll
    for (int r = 0; r < R; ++r) {
      s1[r] = 0.f;
      s2[r] = 0.f;
#pragma unroll
      for (int j = 0; j < VPT; ++j) {
        float xf[8], df[8], gf[8];
        unpack<DT_BF16>(cur.x[r][j], xf);
        unpack<DT_BF16>(cur.d[r][j], df);
        unpack<DT_BF16>(g[j], gf);
#pragma unroll
        for (int k = 0; k < 8; ++k) {
          const float dg = df[k] * gf[k];
          s1[r] += dg;
          s2[r] += dg * ((xf[k] - cur.mu[r]) * cur.rs[r]);
        }
      }
    }
    Rows next;
    if (AHEAD) load(next, row0 + step);   // on its way behind the exchange, the arithmetic and the stores
#pragma unroll
    for (int r = 0; r < R; ++r) {
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) {
        s1[r] += __shfl_xor_sync(0xffffffffu, s1[r], o);
        s2[r] += __shfl_xor_sync(0xffffffffu, s2[r], o);
      }
    }
    if (gw > 1) {
      if (lane == 0) {
#pragma unroll
        for (int r = 0; r < R; ++r) stat[parity][warp][r] = make_float2(s1[r], s2[r]);
      }
      // the other parity's slots are not written again before every warp of the group has passed this barrier once more
      asm volatile("bar.sync %0, %1;" ::"r"(group + 1), "r"(width) : "memory");
#pragma unroll
      for (int r = 0; r < R; ++r) {
        s1[r] = 0.f;
        s2[r] = 0.f;
        for (int w = 0; w < gw; ++w) {
          const float2 p = stat[parity][group * gw + w][r];
          s1[r] += p.x;
          s2[r] += p.y;
        }
      }
    }
#pragma unroll
    for (int r = 0; r < R; ++r) {
      const float m1 = s1[r] * inv_d, m2 = s2[r] * inv_d;
#pragma unroll
      for (int j = 0; j < VPT; ++j) {
        float xf[8], df[8], gf[8], rf[8], of[8];
        unpack<DT_BF16>(cur.x[r][j], xf);
        unpack<DT_BF16>(cur.d[r][j], df);
        unpack<DT_BF16>(g[j], gf);
        if (EXTRA) unpack<DT_BF16>(cur.r[EXTRA ? r : 0][j], rf);
#pragma unroll
        for (int k = 0; k < 8; ++k) {
          const float xh = (xf[k] - cur.mu[r]) * cur.rs[r];
          of[k] = cur.rs[r] * (df[k] * gf[k] - m1 - xh * m2);
          if (EXTRA) of[k] += rf[k];
          ag[j][k] += df[k] * xh;
          ab[j][k] += df[k];
          if (EXTRA) ac[EXTRA ? j : 0][k] += of[k];
        }
        if (row0 + r < rows && tid + j * width < nvec) st16(dx + (row0 + r) * D + (tid + j * width) * 8, pack<DT_BF16>(of));
      }
    }
    if (AHEAD) cur = next;
  }
  const int arrays = EXTRA && part_c ? 3 : 2;
#pragma unroll
  for (int j = 0; j < VPT; ++j) {
    const int v = tid + j * width;
    if (v >= nvec) continue;
#pragma unroll
    for (int a = 0; a < (EXTRA ? 3 : 2); ++a) {
      if (a >= arrays) continue;
      const float* f = a == 0 ? ag[j] : a == 1 ? ab[j] : ac[EXTRA ? j : 0];
      float* dst = groups > 1 ? group_sums + (group * 3 + a) * D + v * 8
                              : (a == 0 ? part_g : a == 1 ? part_b : part_c) + static_cast<long long>(blockIdx.x) * D + v * 8;
      *reinterpret_cast<float4*>(dst) = make_float4(f[0], f[1], f[2], f[3]);
      *reinterpret_cast<float4*>(dst + 4) = make_float4(f[4], f[5], f[6], f[7]);
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

int launchLayerNormFwd(const void* x, const void* delta, void* sum_out, const void* gamma, const void* beta, void* y, float* mean,
                       float* rstd, long long rows, int D, float eps, cudaStream_t stream) {
  if (rows <= 0) return 0;
  if (D % 8 || D > 8192 || (delta && !sum_out) || !aligned16({x, delta, sum_out, gamma, beta, y})) return static_cast<int>(cudaErrorInvalidValue);
  auto X = static_cast<const __nv_bfloat16*>(x); auto G = static_cast<const __nv_bfloat16*>(gamma);
  auto B = static_cast<const __nv_bfloat16*>(beta); auto Y = static_cast<__nv_bfloat16*>(y);
  auto DL = static_cast<const __nv_bfloat16*>(delta); auto S = static_cast<__nv_bfloat16*>(sum_out);
  const int nvec = D / 8;
  int gw = (nvec + 127) / 128, vpt = gw > 1 ? 4 : (nvec + 31) / 32;
  // Up to four million values a thread takes one vector: its chain is the shorter (24 x 2048 9 -> 8 us, 1531 x 2048 equal by itself), and
  // with 40 registers per thread a CTA finds room beside one of a GEMM, to be in its place when that ends.
  if (rows * D <= 4ll << 20 && nvec <= 256) {
    gw = (nvec + 31) / 32;
    vpt = 1;
  }
  // as many rows per CTA as 256 threads hold, fewer where the rows would then leave SMs without work
  int groups = 8 / gw;
  while (groups > 1 && (rows + groups - 1) / groups < deviceSmCount()) groups /= 2;
  const unsigned grid = static_cast<unsigned>((rows + groups - 1) / groups);
  auto go = [&](auto kern) {
    return static_cast<int>(launchOverlapped(kern, dim3(grid), dim3(groups * gw * 32), 0, stream, 1, X, DL, S, G, B, Y, mean, rstd, rows, D, eps, gw));
  };
  return vpt == 1 ? go(ln_fwd_kernel<1>) : vpt == 2 ? go(ln_fwd_kernel<2>) : vpt == 3 ? go(ln_fwd_kernel<3>) : go(ln_fwd_kernel<4>);
}

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
  // VPT vectors per thread, R rows per trip, `sms` CTAs resident per SM
  auto go = [&](auto kern, int vpt, int r, int sms) {
    const int gw = (D / 8 + 32 * vpt - 1) / (32 * vpt), groups = 8 / gw;
    const long long want = (rows + static_cast<long long>(groups) * r - 1) / (static_cast<long long>(groups) * r);
    const int limit = deviceSmCount() * sms < most ? deviceSmCount() * sms : most;
    nparts = static_cast<int>(want < limit ? want : limit);
    const size_t smem = groups > 1 ? static_cast<size_t>(groups) * 3 * D * sizeof(float) : 0;         // at most 24 KiB
    return static_cast<int>(launchOverlapped(kern, dim3(nparts), dim3(groups * gw * 32), smem, stream, 1, static_cast<const __nv_bfloat16*>(dy),
                                             static_cast<const __nv_bfloat16*>(x), static_cast<const __nv_bfloat16*>(gamma), mean, rstd,
                                             static_cast<const __nv_bfloat16*>(dres), static_cast<__nv_bfloat16*>(dx), pg, pb, pc, rows, D, gw));
  };
  int e;
  if (dres || dcolsum)
    e = D <= 2048 ? go(ln_bwd_kernel<1, 4, true, true, 1>, 1, 4, 1) : D <= 4096 ? go(ln_bwd_kernel<2, 2, true, true, 1>, 2, 2, 1)
                                                                                : go(ln_bwd_kernel<4, 1, true, false, 1>, 4, 1, 1);
  else
    e = D <= 2048 ? go(ln_bwd_kernel<1, 2, false, true, 2>, 1, 2, 2) : D <= 4096 ? go(ln_bwd_kernel<2, 2, false, true, 1>, 2, 2, 1)
                                                                                 : go(ln_bwd_kernel<4, 1, false, true, 1>, 4, 1, 1);
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
