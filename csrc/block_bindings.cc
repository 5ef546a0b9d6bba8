// The two halves of a pre-norm transformer block around its attention, forward and backward, each as one call that issues the half's
// launches: norm and QKV projection before it; projection, norm and MLP behind it.  The kernels and their order are those of the layers
// called one by one; what is saved is the caller's way from one launch to the next.  Pointers in, nothing allocated here; weight
// gradients are left to the caller, who knows where they go and who waits for them.
#include <pybind11/pybind11.h>
#include <pybind11/stl.h>

#include <array>
#include <stdexcept>
#include <string>

#include "kernels/elementwise_api.h"
#include "kernels/gemm_api.h"

namespace py = pybind11;
using namespace pccl;

namespace {

template <class T = void>
T* at(uint64_t address) { return reinterpret_cast<T*>(address); }

void check(int err, const char* what) {
  if (err != 0) throw std::runtime_error(std::string(what) + ": " + cudaErrorName(err) + " " + gemmLastError());
}

struct Launch {
  long long rows;
  uint32_t flags;           // GEMM_PAIR or GEMM_SKINNY: the form of the products over `rows`
  uint32_t* status;
  cudaStream_t stream;
  Launch(long long r, uint32_t f, uint64_t st, uint64_t s) : rows(r), flags(f), status(at<uint32_t>(st)), stream(at<CUstream_st>(s)) {}

  // out[rows, n] = a[rows, k] * w[n, k]^T + bias
  void linear(uint64_t a, long long lda, uint64_t w, uint64_t bias, uint64_t out, int n, int k) const {
    check(gemmBf16(at(a), lda, at(w), k, at(out), n, static_cast<int>(rows), n, k, flags | GEMM_BIAS, at(bias), nullptr, 0, status, stream), "linear");
  }
  // pre[rows, n] = the same, act = gelu_tanh of that.  Only a backward pass reads `pre`: without one it may be 0 and is not written (1531 rows
  // of a 2048 x 8192 layer: half of the 50 MB that the epilogue stores; 41.8 -> 37.7 us).
  void linearGelu(uint64_t a, long long lda, uint64_t w, uint64_t bias, uint64_t pre, uint64_t act, int n, int k) const {
    check(gemmBf16(at(a), lda, at(w), k, at(pre ? pre : act), n, static_cast<int>(rows), n, k, flags | GEMM_BIAS | (pre ? GEMM_GELU : GEMM_GELU_INPLACE),
                   at(bias), at(pre ? act : 0), 0, status, stream), "linear and gelu");
  }
  // out[rows, k] = dy[rows, n] * w[n, k]
  void linearBackward(uint64_t dy, uint64_t w, uint64_t out, int n, int k) const {
    check(gemmBf16(at(dy), n, at(w), k, at(out), k, static_cast<int>(rows), k, n, flags | GEMM_B_MN, nullptr, nullptr, 0, status, stream),
          "linear backward");
  }
  // `stats` (or 0): fp32 [2, rows], means and reciprocal deviations
  void norm(uint64_t x, uint64_t delta, uint64_t sum, uint64_t gamma, uint64_t beta, uint64_t y, uint64_t stats, int D, float eps) const {
    check(launchLayerNormFwd(at(x), at(delta), at(sum), at(gamma), at(beta), at(y), at<float>(stats), stats ? at<float>(stats) + rows : nullptr, rows, D, eps,
                             stream), "norm");
  }
  void normBackward(uint64_t dy, uint64_t x, uint64_t gamma, uint64_t stats, uint64_t dres, uint64_t dx, uint64_t dg, uint64_t db, uint64_t dc,
                    uint64_t parts, int D) const {
    check(launchLayerNormBwd(at(dy), at(x), at(gamma), at<float>(stats), at<float>(stats) + rows, at(dres), at(dx), at(dg), at(db), at(dc),
                             at<float>(parts), rows, D, stream), "norm backward");
  }
};

}  // namespace

void bindBlock(py::module_& m) {
  // s = x + delta (delta may be 0: s is x), h = norm(s), qkv = h Wqkv^T + b
  m.def("block_attn_in", [](uint64_t x, uint64_t delta, uint64_t sum, uint64_t gamma, uint64_t beta, float eps, uint64_t h, uint64_t stats, uint64_t w,
                            uint64_t bias, uint64_t qkv, long long rows, int D, uint32_t flags, uint64_t status, uint64_t stream) {
    const Launch l(rows, flags, status, stream);
    l.norm(x, delta, sum, gamma, beta, h, stats, D, eps);
    l.linear(h, D, w, bias, qkv, 3 * D, D);
  });
  // d = a Wp^T + bp, s = x + d, h = norm(s), pre = h W1^T + b1 (0: not kept), act = gelu(pre), out = act W2^T + b2
  m.def("block_mlp_out", [](uint64_t a, long long lda, uint64_t wp, uint64_t bp, uint64_t d, uint64_t x, uint64_t sum, uint64_t gamma, uint64_t beta,
                            float eps, uint64_t h, uint64_t stats, uint64_t w1, uint64_t b1, uint64_t pre, uint64_t act, uint64_t w2, uint64_t b2,
                            uint64_t out, long long rows, int D, int F, uint32_t flags, uint64_t status, uint64_t stream) {
    const Launch l(rows, flags, status, stream);
    l.linear(a, lda, wp, bp, d, D, D);
    l.norm(x, d, sum, gamma, beta, h, stats, D, eps);
    l.linearGelu(h, D, w1, b1, pre, act, F, D);
    l.linear(act, F, w2, b2, out, D, F);
  });
  // The second half backward, without its weight gradients: dpre = (dz W2) gelu'(pre) with its column sums (bf16 [F]; `parts` fp32
  // [ceil(rows / 32), F]), dh = dpre W1, dx = norm'(dh) + dres with the norm's gradients and the column sums dc of dx, da = dx Wp
  m.def("block_mlp_out_bwd", [](uint64_t dz, long long ld_dz, uint64_t w2, uint64_t pre, uint64_t parts, uint64_t colsum, uint64_t dpre, uint64_t w1,
                                uint64_t dh, uint64_t s, uint64_t gamma, uint64_t stats, uint64_t dres, uint64_t dx, uint64_t dg, uint64_t db, uint64_t dc,
                                uint64_t ln_parts, uint64_t wp, uint64_t da, long long rows, int D, int F, uint32_t flags, uint64_t status,
                                uint64_t stream) {
    const Launch l(rows, flags, status, stream);
    check(gemmBf16Dgelu(at(dz), ld_dz, at(w2), F, at(dpre), F, at(pre), ColSum{at<float>(parts), at(colsum), false}, static_cast<int>(rows), F, D, GEMM_B_MN,
                        0, l.status, l.stream), "gelu backward");
    l.linearBackward(dpre, w1, dh, F, D);
    l.normBackward(dh, s, gamma, stats, dres, dx, dg, db, dc, ln_parts, D);
    l.linearBackward(dx, wp, da, D, D);
  });
  // The first half backward, without its weight gradient: dqkv = pack(dq, dk, dv) with its column sums, dh = dqkv Wqkv,
  // dx = norm'(dh) + dres (0: none) with the norm's gradients and the column sums dc of dx (0: none)
  m.def("block_attn_in_bwd", [](const std::array<uint64_t, 3>& grads, const std::array<long long, 9>& strides, uint64_t dqkv, int batch, int seq, int heads,
                                int hd, uint64_t colsum, uint64_t parts, uint64_t w, uint64_t dh, uint64_t s, uint64_t gamma, uint64_t stats, uint64_t dres,
                                uint64_t dx, uint64_t dg, uint64_t db, uint64_t dc, uint64_t ln_parts, uint32_t flags, uint64_t status,
                                uint64_t stream) {
    const int D = heads * hd;
    const Launch l(static_cast<long long>(batch) * seq, flags, status, stream);
    const void* g[3] = {at(grads[0]), at(grads[1]), at(grads[2])};
    check(launchQkvPack(g, strides.data(), at(dqkv), batch, seq, heads, hd, at(colsum), at<float>(parts), l.stream), "qkv pack");
    l.linearBackward(dqkv, w, dh, 3 * D, D);
    l.normBackward(dh, s, gamma, stats, dres, dx, dg, db, dc, ln_parts, D);
  });
}
