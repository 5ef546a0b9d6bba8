// Element-wise / row-wise kernels of the training path (AdamW, cross-entropy, LayerNorm).  No counterpart in the reference.
// Host entry points of the memory-bound training kernels (elementwise.cu).
#pragma once
#include <cuda_runtime.h>

#include <cstdint>

namespace pccl {

// AdamW step `step` (1-based) on n elements: p/m/v fp32 are updated in place from g * grad_scale,
// and the new parameters are also written as bf16 to p_bf16.
int launchAdamW(float* p, float* m, float* v, const float* g, void* p_bf16, long long n, float lr, float b1, float b2,
                float eps, float wd, int step, float grad_scale, cudaStream_t stream);

// Softmax cross-entropy over bf16 logits [rows, vocab] with row stride ld (multiple of 8):
// loss[row] = logsumexp - logit[target]; the logits are overwritten by
// (softmax - onehot) * grad_scale (rows whose target equals ignore_index get zeros).  Targets must lie in [0, vocab);
// any other value is treated like ignore_index (loss 0, zero gradient, no access outside the row) and, when `status`
// (4 x u32, device, may be null) is given and still clear, recorded there as {ST_BOUNDS, row, target, 0xCE}.
int launchCrossEntropy(void* logits, const long long* targets, float* loss, long long rows, int vocab, long long ld,
                       float grad_scale, long long ignore_index, uint32_t* status, cudaStream_t stream);

// out[b, t] = tok[ids[b, t]] + pos[t] for bf16 tables tok [vocab, D], pos [>= seq, D] (D % 8 == 0, 16-byte aligned); n_ids = batch * seq,
// n_ids * D / 8 < 2^31.
// Negative indices count from the end; one outside the table is a device assertion, as in the index kernels of the framework underneath.
int launchEmbedFwd(const long long* ids, const void* tok, const void* pos, void* out, long long n_ids, int seq, long long vocab, int D,
                   cudaStream_t stream);
// Backward: rows of dy [batch, seq, D] are added to d_tok (bf16 [vocab, D], may be null) and summed over the batch into d_pos (bf16,
// may be null), written or, with `add_pos`, added.
int launchEmbedBwd(const void* dy, const long long* ids, void* d_tok, void* d_pos, int batch, int seq, long long vocab, int D, bool add_pos,
                   cudaStream_t stream);

// LayerNorm over the last dimension D (multiple of 8, <= 8192) of bf16 [rows, D]; mean / rstd are fp32 [rows], or both
// null where no backward pass follows.
// With `delta` (bf16 [rows, D], may be null) the norm is taken of s = x + delta and s is stored to `sum_out`:
// the residual connection of a pre-norm block and the norm in one pass.
//
// How a launch divides its rows: warps per row, 16-byte vectors per thread, rows per CTA, and whether the CTA is one row's by construction (a
// kernel with one barrier; the other one names its barriers at run time and takes all 16, so an SM holds fewer CTAs of it).
// Measured on 148 SMs behind a GEMM that writes the rows (us; a CTA of as many rows as fit / one row per CTA):
//   1531 x 2048 5.6 / 3.8, 1000 x 1536 3.9 / 2.7, 128 x 1536 2.3 / 2.1, 1 x 2560 3.0 / 2.2, 128 x 4096 2.8 / 2.3, 1531 x 3072 6.2 / 5.1, 3000 x
//   2560 9.2 / 6.9, 4096 x 5120 23 / 16, but 300 x 2048 2.4 / 2.4 (with the residual sum 2.6 / 2.9), 300 x 4096 3.2 / 3.8, 2331 x 2048 4.7 / 5.3:
// one row per CTA up to one row per SM and, beyond D = 1024, from more than three on, but not for large inputs of up to 2048 columns.
// One vector per thread (two beyond 2048, three beyond 4096, four beyond 6144) is the shorter chain, which few rows need; four per thread
// leave more rows in flight on an SM: from 7 Mi values on up to D = 5120 (4096 x 3072 11.4 -> 9.5, but 1531 x 4096, 6 Mi, 6.0 -> 6.6).
// Eight warps of two vectors fit an SM six times: the seventh and eighth row of an SM would be a second round (1000 x 4096 4.5 / 4.8).
// Up to eight rows per SM eight warps spread more evenly than the five to seven that narrower rows need (800 x 1032 3.7 -> 3.4).
struct LayerNormFwdForm { int warps, vectors, rows; bool one_row; };
LayerNormFwdForm layerNormFwdForm(long long rows, int D, int sms);
int launchLayerNormFwd(const void* x, const void* delta, void* sum_out, const void* gamma, const void* beta, void* y, float* mean,
                       float* rstd, long long rows, int D, float eps, cudaStream_t stream);
// Backward: dx bf16 [rows, D] = d(norm input) + dres (bf16 [rows, D], may be null: the gradient on the residual stream);
// dgamma / dbeta bf16 [D]; dcolsum (bf16 [D], may be null) receives the column sums of dx, which is the bias gradient of
// the linear layer that fed the residual sum.  `x` is the norm's input (the stored sum when forward had a delta).
// `partials` is fp32 scratch of 3 * layerNormBwdParts(rows) * D elements.
int layerNormBwdParts(long long rows);
// Whether a backward pass with a residual gradient or column sums takes its rows through the ring in shared memory: from 16 rows per SM on
// beyond 2048 columns, from 7 on beyond 4096 (the kernel has both sides' times).
bool layerNormBwdRing(long long rows, int D, int sms);
int launchLayerNormBwd(const void* dy, const void* x, const void* gamma, const float* mean, const float* rstd, const void* dres, void* dx,
                       void* dgamma, void* dbeta, void* dcolsum, float* partials, long long rows, int D, cudaStream_t stream);

// out[n] = sum over rows of x[row, n] for bf16 x [rows, N] with row stride ld (elements, multiple of 8); N a multiple of 8.
// `partials`: fp32 scratch of colSumParts(rows) * N elements.
int colSumParts(long long rows);
int launchColSum(const void* x, long long ld, long long rows, int N, void* out_bf16, float* partials, cudaStream_t stream);

// Column sums that a GEMM epilogue takes of its output: it leaves the sum of every 32 rows in `parts` (fp32 [ceil(M / 32), N]), and
// launchColSumParts adds those up in row order, so a run repeats itself exactly (atomic additions from the epilogue did not).
// `out`: fp32 [N] that grows by the sums, or bf16 [N] that is written.  No sums if `out` is null.
struct ColSum {
  float* parts;
  void* out;
  bool f32;
};
int launchColSumParts(const ColSum& c, int M, int N, cudaStream_t stream);

// Gradients of q, k, v (grads[3], bf16 [batch, heads, seq, hd] with strides[3 i ..] = batch, head, position in elements, multiples
// of 8; the last dimension contiguous) packed into out [batch * seq, 3, heads, hd], and its column sums as bf16 [3 * heads * hd].
// `partials`: fp32 scratch of colSumParts(batch * seq) * 3 * heads * hd elements.
int launchQkvPack(const void* const* grads, const long long* strides, void* out, int batch, int seq, int heads, int hd, void* colsum_bf16,
                  float* partials, cudaStream_t stream);

}  // namespace pccl
