"""tcgen05 GEMM against an fp32 PyTorch reference of the same op."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _ref(a, b, a_t, b_t):
    A = a.float().t() if a_t else a.float()
    B = b.float() if b_t else b.float().t()
    return A @ B


def _rand(shape, seed, scale=1.0):
    g = torch.Generator(device="cuda").manual_seed(seed)
    return (torch.randn(shape, generator=g, device="cuda") * scale).bfloat16()


@pytest.mark.parametrize("M,N,K", [(128, 256, 64), (256, 512, 256), (384, 768, 1024), (1000, 520, 200), (72, 40, 136)])
@pytest.mark.parametrize("a_t,b_t", [(False, False), (False, True), (True, True), (True, False)])
def test_gemm_matches_fp32_reference(M, N, K, a_t, b_t):
    from pccl_b200.ops import gemm, check_status
    a = _rand((K, M) if a_t else (M, K), 1)
    b = _rand((K, N) if b_t else (N, K), 2)
    out = gemm(a, b, a_t=a_t, b_t=b_t)
    check_status("gemm")
    ref = _ref(a, b, a_t, b_t)
    err = (out.float() - ref).abs().max().item()
    tol = 2e-2 * (K ** 0.5) * 0.25 + 1e-2 * ref.abs().max().item()
    assert err <= tol, f"max err {err} > {tol}"
    # fp32 output is compared tightly: products of bf16 are exact in fp32, only the sum order differs
    out32 = gemm(a, b, a_t=a_t, b_t=b_t, out_dtype=torch.float32)
    assert (out32 - ref).abs().max().item() <= 1e-3 * max(1.0, ref.abs().max().item())


def test_gemm_epilogues():
    from pccl_b200.ops import gemm, check_status
    M, N, K = 512, 1024, 512
    a, b = _rand((M, K), 3), _rand((N, K), 4, 0.05)
    bias = _rand((N,), 5)
    act = torch.empty((M, N), dtype=torch.bfloat16, device="cuda")
    pre = gemm(a, b, bias=bias, gelu_out=act)
    check_status("gemm")
    ref = a.float() @ b.float().t() + bias.float()
    assert (pre.float() - ref).abs().max().item() < 0.05
    ref_act = torch.nn.functional.gelu(ref, approximate="tanh")    # the kernel applies GELU before rounding
    assert ((act.float() - ref_act).abs() <= 0.01 + 0.01 * ref_act.abs()).all()
    acc = torch.ones((M, N), dtype=torch.float32, device="cuda")
    gemm(a, b, out=acc, accumulate=True)
    assert (acc - (a.float() @ b.float().t() + 1)).abs().max().item() < 1e-2


def test_gemm_padded_leading_dimension():
    from pccl_b200.ops import gemm
    M, N, K = 300, 1001, 264                     # N not a multiple of 8: row stride is padded
    a, b = _rand((M, K), 6), _rand((N, K), 7)
    out = gemm(a, b)
    assert out.shape == (M, N) and out.stride(0) == 1008
    assert (out.float() - a.float() @ b.float().t()).abs().max().item() < 0.5
    # consume it again as a K-padded operand
    w = _rand((128, N), 8, 0.1)
    wp = torch.zeros((128, 1008), dtype=torch.bfloat16, device="cuda")[:, :N]
    wp.copy_(w)
    y = gemm(out, wp)
    assert (y.float() - out.float() @ w.float().t()).abs().max().item() < 1.0


@pytest.mark.parametrize("M,N,K", [(256, 256, 64), (512, 768, 512), (1000, 520, 200), (72, 40, 136), (2048, 1024, 1024)])
@pytest.mark.parametrize("a_t,b_t", [(False, False), (False, True), (True, True), (True, False)])
def test_cta_pair_gemm_matches_fp32_reference(M, N, K, a_t, b_t):
    """cta_group::2 kernel: two CTAs per 256 x 256 tile."""
    from pccl_b200.ops import gemm, check_status
    a = _rand((K, M) if a_t else (M, K), 11)
    b = _rand((K, N) if b_t else (N, K), 12)
    out32 = gemm(a, b, a_t=a_t, b_t=b_t, out_dtype=torch.float32, pair=True)
    check_status("pair gemm")
    ref = _ref(a, b, a_t, b_t)
    assert (out32 - ref).abs().max().item() <= 1e-3 * max(1.0, ref.abs().max().item())
    bias = _rand((N,), 13)
    out = gemm(a, b, a_t=a_t, b_t=b_t, bias=bias, pair=True)
    assert (out.float() - (ref + bias.float())).abs().max().item() <= 0.02 * max(1.0, ref.abs().max().item())


@pytest.mark.parametrize("M,N,K", [(128, 256, 128), (256, 512, 1024), (384, 768, 2048), (1000, 640, 512), (72, 128, 256)])
def test_fp8_block_scaled_gemm_matches_fp32_reference_of_the_quantised_operands(M, N, K):
    from pccl_b200.ops import check_status
    from pccl_b200.ops.gemm import dequant_blocks, dequant_rows, gemm_fp8, quant_blocks, quant_rows
    a = _rand((M, K), 3)
    w = _rand((N, K), 4, scale=0.02)
    # per-block magnitudes that differ by orders of magnitude, so that a wrong scale index shows
    a = (a.float() * torch.logspace(-2, 2, K // 128, device="cuda").repeat_interleave(128)[None, :]).bfloat16()
    aq, a_s = quant_rows(a)
    wq, w_s = quant_blocks(w)
    out32 = gemm_fp8(aq, a_s, wq, w_s, out_dtype=torch.float32)
    check_status("gemm_fp8")
    ref = dequant_rows(aq, a_s) @ dequant_blocks(wq, w_s).t()
    scale = max(1.0, ref.abs().max().item())
    # the kernel's sum is exact products of e4m3 values accumulated in fp32: only the order differs
    assert (out32 - ref).abs().max().item() <= 2e-3 * scale
    out = gemm_fp8(aq, a_s, wq, w_s)
    assert (out.float() - ref).abs().max().item() <= 1e-2 * scale
    # and the quantised product stays close to the bf16 one
    full = a.float() @ w.float().t()
    assert (ref - full).abs().max().item() <= 0.08 * full.abs().max().item()


def test_fp8_gemm_bias_and_accumulate():
    from pccl_b200.ops import check_status
    from pccl_b200.ops.gemm import dequant_blocks, dequant_rows, gemm_fp8, quant_blocks, quant_rows
    M, N, K = 256, 384, 512
    aq, a_s = quant_rows(_rand((M, K), 5))
    wq, w_s = quant_blocks(_rand((N, K), 6, scale=0.05))
    bias = _rand((N,), 7)
    ref = dequant_rows(aq, a_s) @ dequant_blocks(wq, w_s).t()
    out = torch.ones((M, N), device="cuda", dtype=torch.float32)
    gemm_fp8(aq, a_s, wq, w_s, out=out, bias=bias, accumulate=True)
    check_status("gemm_fp8")
    assert (out - (ref + bias.float()[None, :] + 1.0)).abs().max().item() <= 2e-3 * max(1.0, ref.abs().max().item())


def test_mx_quantisers_give_power_of_two_scales_that_cover_the_block():
    from pccl_b200.ops.gemm import dequant_rows, quant_blocks_mx, quant_rows_mx, ue8m0_to_float
    x = _rand((200, 512), 11, scale=3.0)
    q, s = quant_rows_mx(x)
    sc = ue8m0_to_float(s)
    amax = x.float().view(200, 4, 128).abs().amax(-1)
    assert torch.all(sc * 448.0 >= amax) and torch.all(sc * 224.0 < amax.clamp_min(1e-30) * 1.0000001)
    back = dequant_rows(q, sc)
    assert (back - x.float()).abs().max().item() <= 0.07 * x.float().abs().max().item()
    w = _rand((256, 384), 12, scale=0.02)
    qw, sw = quant_blocks_mx(w)
    amaxw = w.float().view(2, 128, 3, 128).abs().amax((1, 3))
    assert torch.all(ue8m0_to_float(sw) * 448.0 >= amaxw)


@pytest.mark.parametrize("M,N,K", [(128, 128, 128), (128, 256, 512), (256, 512, 1024), (384, 768, 2048), (1000, 640, 640), (72, 128, 256)])
def test_mx_fp8_gemm_matches_fp32_reference_of_the_quantised_operands(M, N, K):
    from pccl_b200.ops import check_status
    from pccl_b200.ops.gemm import dequant_blocks, dequant_rows, gemm_mx8, quant_blocks_mx, quant_rows_mx, ue8m0_to_float
    a = _rand((M, K), 13)
    w = _rand((N, K), 14, scale=0.02)
    # magnitudes that differ per K block AND per row group / column block, so that a wrong scale index shows
    a = (a.float() * torch.logspace(-2, 2, K // 128, device="cuda").repeat_interleave(128)[None, :]
         * (1.0 + (torch.arange(M, device="cuda") // 32 % 4).float())[:, None]).bfloat16()
    w = (w.float() * (1.0 + 3.0 * (torch.arange(N, device="cuda") // 128).float())[:, None]).bfloat16()
    aq, a_s = quant_rows_mx(a)
    wq, w_s = quant_blocks_mx(w)
    out32 = gemm_mx8(aq, a_s, wq, w_s, out_dtype=torch.float32)
    check_status("gemm_mx8")
    ref = dequant_rows(aq, ue8m0_to_float(a_s)) @ dequant_blocks(wq, ue8m0_to_float(w_s)).t()
    scale = max(1.0, ref.abs().max().item())
    assert (out32 - ref).abs().max().item() <= 2e-3 * scale
    out = gemm_mx8(aq, a_s, wq, w_s)
    assert (out.float() - ref).abs().max().item() <= 1e-2 * scale


def test_gemm_residual_epilogue_adds_the_residual_stream():
    """out = a @ b.T + bias + residual in the GEMM epilogue (full and ragged tiles)."""
    from pccl_b200.ops import gemm, check_status
    for (M, N, K) in [(512, 1024, 256), (300, 264, 128)]:
        a, b = _rand((M, K), 21), _rand((N, K), 22, 0.05)
        bias, res = _rand((N,), 23), _rand((M, N), 24)
        out = gemm(a, b, bias=bias, residual=res)
        check_status("gemm residual")
        ref = a.float() @ b.float().t() + bias.float() + res.float()
        assert (out.float() - ref).abs().max().item() <= 2e-2 * max(1.0, ref.abs().max().item())


# The CTA-pair kernel picks its tile width per launch: every width, with rows and columns that end inside a tile and inside a
# 32-column strip.
@pytest.mark.parametrize("M,N,K,width", [(257, 40, 72, 32), (300, 1416, 200, 64), (200, 4808, 72, 96), (2331, 776, 264, 128), (4096, 3576, 128, 160),
                                         (1999, 1416, 328, 160), (1531, 2056, 136, 192), (1531, 6152, 64, 192), (700, 4664, 136, 224), (700, 5480, 72, 256)])
@pytest.mark.parametrize("a_t,b_t", [(False, False), (False, True), (True, True)])
def test_cta_pair_gemm_tile_widths(M, N, K, width, a_t, b_t):
    from pccl_b200._native import C
    from pccl_b200.ops import gemm, check_status
    assert C.gemm_pair_tile_n((M + 255) // 256, N, 0, 0, 74) == width          # 148 SMs
    if a_t:
        M = (M + 7) // 8 * 8
    a = _rand((K, M) if a_t else (M, K), 61)
    b = _rand((K, N) if b_t else (N, K), 62)
    ref = _ref(a, b, a_t, b_t)
    out32 = gemm(a, b, a_t=a_t, b_t=b_t, out_dtype=torch.float32, pair=True)
    bias = _rand((N,), 63)
    act = torch.full((M, N), 7.0, dtype=torch.bfloat16, device="cuda")
    pre = torch.empty_like(act)
    gemm(a, b, a_t=a_t, b_t=b_t, out=pre, bias=bias, gelu_out=act, pair=True)
    check_status("pair gemm widths")
    # fp32 sums of K exact products in another order: K * 2^-24 of the absolute sum, far below 1e-3 of the largest result
    assert (out32 - ref).abs().max().item() <= 1e-3 * max(1.0, ref.abs().max().item())
    full = ref + bias.float()
    assert (pre.float() - full).abs().max().item() <= 2 ** -8 * full.abs().max().item()           # one bf16 rounding
    gelu = torch.nn.functional.gelu(full, approximate="tanh")
    assert ((act.float() - gelu).abs() <= 0.01 + 0.01 * gelu.abs()).all()                            # hardware tanh, then bf16


@pytest.mark.parametrize("M", [1, 40, 1531])
def test_gemm_dgelu_ragged_rows(M):
    from pccl_b200.ops import check_status
    from pccl_b200.ops.gemm import gemm_dgelu
    N, K = 1056, 136
    a, b, pre = _rand((M, K), 64), _rand((K, N), 65, 0.05), _rand((M, N), 66, 1.5)
    sums = torch.zeros(N, dtype=torch.float32, device="cuda")
    out = gemm_dgelu(a, b, pre, b_t=True, colsum=sums)
    check_status("gemm dgelu ragged")
    x = pre.float().requires_grad_(True)
    torch.nn.functional.gelu(x, approximate="tanh").backward(a.float() @ b.float())
    ref = x.grad
    assert (out.float() - ref).abs().max().item() <= 2e-2 * max(1.0, ref.abs().max().item())
    assert (sums - ref.sum(0)).abs().max().item() <= 2e-2 * max(1.0, ref.sum(0).abs().max().item())


@pytest.mark.parametrize("M,N", [(40, 256), (256, 288), (513, 1056), (700, 4672)])            # the last one: tiles of 224 columns
def test_gemm_dgelu_off_the_tiles_is_accurate_on_the_negative_side(M, N):
    """gelu' where 1 - tanh^2 cancels: within the bf16 rounding of every single value, against fp64.  The product is exact (one
    nonzero per row of a), so 2^-8 is the rounding; 1e-4 of |gelu'| <= 1.2 covers the exponential's and the division's error."""
    from pccl_b200.ops import check_status
    from pccl_b200.ops.gemm import gemm_dgelu
    K = 64
    a = torch.zeros((M, K), dtype=torch.bfloat16, device="cuda")
    a[torch.arange(M), torch.arange(M) % K] = 1.0
    b = _rand((K, N), 67)
    pre = (-1.0 - 3.0 * torch.rand((M, N), device="cuda")).bfloat16()
    out = gemm_dgelu(a, b, pre, b_t=True)
    check_status("gemm dgelu accuracy")
    x = pre.double().requires_grad_(True)
    torch.nn.functional.gelu(x, approximate="tanh").backward(a.double() @ b.double())
    assert ((out.double() - x.grad).abs() <= (2 ** -8 + 1e-4) * x.grad.abs() + 1e-7).all()


@pytest.mark.parametrize("M,N", [(1, 32), (31, 96), (33, 256), (2048, 512), (9001, 288)])
def test_gemm_dgelu_column_sums_repeat_exactly(M, N):
    """The bias gradient is the same from run to run, in both forms; fp32 sums of M values in groups of 32 rows, against fp64 sums of
    the values themselves, which differ from the summed ones by one bf16 rounding each."""
    from pccl_b200.ops import check_status
    from pccl_b200.ops.gemm import gemm_dgelu
    K = 64
    a, b, pre = _rand((M, K), 68), _rand((K, N), 69, 0.1), _rand((M, N), 70)
    runs = []
    for _ in range(4):
        f32, b16 = torch.full((N,), 3.0, device="cuda"), torch.full((N,), 9.0, dtype=torch.bfloat16, device="cuda")
        out = gemm_dgelu(a, b, pre, b_t=True, colsum=f32)
        gemm_dgelu(a, b, pre, b_t=True, colsum=b16)
        runs.append((out, f32, b16))
    check_status("gemm dgelu sums")
    for r in runs[1:]:
        assert all(torch.equal(x, y) for x, y in zip(r, runs[0]))
    out, f32, b16 = runs[0]
    want, spread = out.double().sum(0), out.double().abs().sum(0)
    assert ((f32.double() - 3 - want).abs() <= 2 ** -8 * spread + 1e-5).all()
    assert ((b16.double() - want).abs() <= 2 ** -8 * (spread + want.abs()) + 1e-5).all()


@pytest.mark.parametrize("M", [1, 15, 17, 33, 100, 128])
@pytest.mark.parametrize("N,K,splits", [(40, 72, 1), (1001, 200, 1), (512, 2048, 8), (8200, 520, 2), (1001, 1032, 4), (8190, 1096, 4)])
@pytest.mark.parametrize("b_t", [False, True])
def test_few_row_gemm(M, N, K, splits, b_t):
    """Weights on the tile's M side, K split over a cluster of 1, 2, 4 or 8 CTAs, with every epilogue."""
    from pccl_b200._native import C
    from pccl_b200.ops import gemm, check_status
    assert C.gemm_skinny_splits(N, K, 148) == splits
    ld = (N + 7) // 8 * 8
    a = _rand((M, K), 71)
    b = _rand((K, ld), 72)[:, :N] if b_t else _rand((N, K), 72)
    ref = _ref(a, b, False, b_t)
    big = max(1.0, ref.abs().max().item())
    acc = torch.ones((M, ld), dtype=torch.float32, device="cuda")[:, :N]
    gemm(a, b, b_t=b_t, out=acc, accumulate=True)
    bias, res = _rand((N,), 73), _rand((M, ld), 74)[:, :N]
    act = torch.full((M, ld), 9.0, dtype=torch.bfloat16, device="cuda")
    pre = torch.full((M, ld), 9.0, dtype=torch.bfloat16, device="cuda")
    gemm(a, b, b_t=b_t, bias=bias, gelu_out=act[:, :N], out=pre[:, :N])
    out = torch.empty((M, ld), dtype=torch.bfloat16, device="cuda")[:, :N]
    gemm(a, b, b_t=b_t, bias=bias, residual=res, out=out)
    check_status("few-row gemm")
    assert (acc - ref - 1).abs().max().item() <= 1e-3 * big                   # fp32, sums in another order
    full = ref + bias.float()
    assert (pre[:, :N].float() - full).abs().max().item() <= 2 ** -8 * full.abs().max().item()      # one bf16 rounding
    gelu = torch.nn.functional.gelu(full, approximate="tanh")
    assert ((act[:, :N].float() - gelu).abs() <= 0.01 + 0.01 * gelu.abs()).all()
    assert (out.float() - full - res.float()).abs().max().item() <= 2 ** -8 * (full + res.float()).abs().max().item()
    assert (act[:, N:] == 9.0).all() and (pre[:, N:] == 9.0).all()             # nothing past the last column


@pytest.mark.parametrize("b_t", [True, False])
def test_gemm_dgelu_epilogue_and_column_sums(b_t):
    """(a @ op(b)) * gelu_tanh'(pre) with the column sums of the result, against fp32 PyTorch."""
    from pccl_b200.ops import check_status
    from pccl_b200.ops.gemm import gemm_dgelu
    M, N, K = 512, 768, 256
    a = _rand((M, K), 31)
    b = _rand((K, N) if b_t else (N, K), 32, 0.05)
    pre = _rand((M, N), 33, 1.5)
    sums = torch.zeros(N, dtype=torch.float32, device="cuda")
    out = gemm_dgelu(a, b, pre, b_t=b_t, colsum=sums)
    check_status("gemm dgelu")
    prod = a.float() @ (b.float() if b_t else b.float().t())
    x = pre.float().requires_grad_(True)
    torch.nn.functional.gelu(x, approximate="tanh").backward(prod)
    ref = x.grad
    assert (out.float() - ref).abs().max().item() <= 2e-2 * max(1.0, ref.abs().max().item())
    assert (sums - ref.sum(0)).abs().max().item() <= 2e-2 * max(1.0, ref.sum(0).abs().max().item())
    # without column sums the product is the same
    out2 = gemm_dgelu(a, b, pre, b_t=b_t)
    assert torch.equal(out, out2)


@pytest.mark.parametrize("shapes", [((512, 256), (256, 768)), ((304, 520), (1032, 136)), ((2048, 8192), (8192, 2048))])
@pytest.mark.parametrize("out_dtype", [torch.bfloat16, torch.float32])
def test_gemm_dual_two_weight_gradients_one_launch(shapes, out_dtype):
    """Two dW = dy^T x products of one row count as a single launch, fresh and accumulating, against fp32 PyTorch."""
    from pccl_b200.ops import check_status
    from pccl_b200.ops.gemm import gemm_dual
    rows = 1024
    (m0, n0), (m1, n1) = shapes
    dy0, x0 = _rand((rows, m0), 51, 0.1), _rand((rows, n0), 52)
    dy1, x1 = _rand((rows, m1), 53, 0.1), _rand((rows, n1), 54)
    o0 = torch.full((m0, n0), 3.0, dtype=out_dtype, device="cuda")
    o1 = torch.full((m1, n1), -2.0, dtype=out_dtype, device="cuda")
    gemm_dual(dy0, x0, o0, dy1, x1, o1, a_t=True, b_t=True, accumulate1=True)
    check_status("gemm dual")
    r0 = dy0.float().t() @ x0.float()
    r1 = dy1.float().t() @ x1.float() - 2.0
    for got, ref in ((o0, r0), (o1, r1)):
        assert (got.float() - ref).abs().max().item() <= 2e-2 * max(1.0, ref.abs().max().item())
    # the plain (K-major) operand forms go through the same scheduler
    a0, b0 = _rand((m0, 192), 55), _rand((n0, 192), 56)
    a1, b1 = _rand((m1, 192), 57), _rand((n1, 192), 58)
    p0 = torch.empty((m0, n0), dtype=out_dtype, device="cuda")
    p1 = torch.empty((m1, n1), dtype=out_dtype, device="cuda")
    gemm_dual(a0, b0, p0, a1, b1, p1)
    check_status("gemm dual k-major")
    for got, ref in ((p0, a0.float() @ b0.float().t()), (p1, a1.float() @ b1.float().t())):
        assert (got.float() - ref).abs().max().item() <= 2e-2 * max(1.0, ref.abs().max().item())


@pytest.mark.parametrize("rows,N", [(16384, 2048), (1000, 520), (37, 8)])
def test_colsum_kernel_matches_torch(rows, N):
    from pccl_b200.ops.elementwise import colsum
    x = _rand((rows, N), 41)
    got = colsum(x)
    ref = x.float().sum(0)
    assert (got.float() - ref).abs().max().item() <= 1e-2 * max(1.0, ref.abs().max().item())
    view = _rand((rows, N + 24), 42)[:, 8:8 + N] if N % 8 == 0 and N > 8 else None     # a column slice of a wider buffer
    if view is not None and view.data_ptr() % 16 == 0:
        assert (colsum(view).float() - view.float().sum(0)).abs().max().item() <= 1e-2 * max(1.0, view.float().sum(0).abs().max().item())


@pytest.mark.parametrize("M,N,width", [(1, 40, 160), (33, 40, 32), (130, 1000, 32), (300, 4104, 96), (1531, 3584, 160), (2000, 520, 64), (700, 4104, 192),
                                       (1531, 2400, 224), (19000, 232, 128), (9000, 448, 224)])
def test_mx8_tile_widths(M, N, width):
    """Sizes over which the launch picks tiles of 32 ... 224 columns, with ragged last tiles and scale blocks that a tile straddles.
    fp32 output against the product of the dequantised operands: the sums differ in their order only."""
    from pccl_b200._native import C
    from pccl_b200.ops import check_status
    from pccl_b200.ops.gemm import dequant_rows, gemm_mx8, quant_rows_mx, ue8m0_to_float
    assert C.gemm_mx8_tile_n(M, N, 148) == width
    K = 384
    a, w = _rand((M, K), 81), _rand((N, K), 82)
    aq, a_s = quant_rows_mx(a)
    wq, w_rows = quant_rows_mx(w)
    w_s = w_rows[::128].contiguous()                      # one scale byte per 128 rows: any byte is as good as another here
    out = gemm_mx8(aq, a_s, wq, w_s, out_dtype=torch.float32)
    check_status("gemm_mx8")
    af = dequant_rows(aq, ue8m0_to_float(a_s))
    wf = wq.view(torch.float8_e4m3fn).float() * ue8m0_to_float(w_s).repeat_interleave(128, 1).repeat_interleave(128, 0)[:N]
    ref = af.double() @ wf.double().t()
    assert (out.double() - ref).abs().max().item() <= 2e-3 * max(1.0, ref.abs().max().item())      # a wrong scale or tile is off by O(1)


@pytest.mark.parametrize("out_dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("M,N", [(40, 72), (300, 1000)])
def test_fp8_gelu_in_every_column(M, N, out_dtype):
    """GELU on the output reaches the columns past the last whole strip of 32 and fp32 outputs as well; against the same product
    without it (hardware tanh: 2^-11 of the value, 1e-3 on the flat side), and one bf16 rounding."""
    from pccl_b200.ops import check_status
    from pccl_b200.ops.gemm import gemm_fp8, gemm_mx8, quant_blocks, quant_blocks_mx, quant_rows, quant_rows_mx
    K = 256
    a, w = _rand((M, K), 91), _rand(((N + 127) // 128 * 128, K), 92, 0.1)
    for g, qr, qb in ((gemm_fp8, quant_rows, quant_blocks), (gemm_mx8, quant_rows_mx, quant_blocks_mx)):
        aq, a_s = qr(a)
        wq, w_s = qb(w)
        plain = g(aq, a_s, wq[:N], w_s, out_dtype=torch.float32)
        act = g(aq, a_s, wq[:N], w_s, out_dtype=out_dtype, gelu_inplace=True)
        check_status("fp8 gelu")
        want = torch.nn.functional.gelu(plain.double(), approximate="tanh")
        assert ((act.double() - want).abs() <= (2 ** -8 if out_dtype is torch.bfloat16 else 2 ** -10) * want.abs() + 1.5e-3 * plain.abs()).all()


@pytest.mark.parametrize("M,pair", [(40, None), (200, False), (200, True)])
def test_gemm_second_output_off_the_16_byte_boundaries(M, pair):
    """A second output that starts anywhere (its rows are strided like out's) gets what an aligned one gets."""
    from pccl_b200.ops import check_status, gemm
    N, K, ld = 96, 64, 104
    a, w = _rand((M, K), 93), _rand((N, K), 94, 0.2)
    def strided(shift):
        return torch.zeros((M, ld), dtype=torch.bfloat16, device="cuda").view(-1)[shift:shift + M * ld - 8].as_strided((M, N), (ld, 1))
    got = []
    for shift in (0, 1, 4):
        act, pre = strided(shift), strided(0)
        gemm(a, w, gelu_out=act, out=pre, pair=pair)
        got.append([pre.clone(), act.clone()])
    check_status("second output")
    assert all(torch.equal(x, y) for g in got[1:] for x, y in zip(g, got[0]))
    ref = a.double() @ w.double().t()
    assert ((got[0][0].double() - ref).abs() <= 2 ** -8 * ref.abs() + 1e-4).all()


@pytest.mark.parametrize("M,N,K", [(1, 8, 128), (127, 136, 256), (129, 264, 640), (260, 1000, 1152), (3000, 128, 384)])
def test_fp8_gemm_at_the_edges_of_its_tiles(M, N, K):
    """Ragged rows and columns around 128, one to nine K blocks (four accumulators are taken in turn), scales that differ per block;
    fp32 output against the product of the dequantised operands (2e-3, as for the other fp8 forms)."""
    from pccl_b200.ops import check_status
    from pccl_b200.ops.gemm import dequant_rows, gemm_fp8, quant_rows
    a = (_rand((M, K), 91).float() * torch.logspace(-1, 1, K // 128, device="cuda").repeat_interleave(128)).bfloat16()
    wq, w_rows = quant_rows(_rand((N, K), 92))
    aq, a_s = quant_rows(a)
    w_s = (w_rows[::128] * (1.0 + torch.arange((N + 127) // 128, device="cuda")[:, None])).contiguous()
    out = gemm_fp8(aq, a_s, wq, w_s, out_dtype=torch.float32)
    check_status("gemm_fp8")
    wf = wq.view(torch.float8_e4m3fn).double() * w_s.double().repeat_interleave(128, 1).repeat_interleave(128, 0)[:N]
    ref = dequant_rows(aq, a_s).double() @ wf.t()
    assert (out.double() - ref).abs().max().item() <= 2e-3 * max(1.0, ref.abs().max().item())


@pytest.mark.parametrize("K", [512, 640, 896, 1024, 1152, 1408, 1536])
@pytest.mark.parametrize("shift,stride", [(0, 4), (0, 12), (1, 12), (0, 9)])
def test_fp8_gemm_row_scales_of_any_stride(K, shift, stride):
    """Row scales are read four K blocks at a time where their rows allow it and there are eight blocks: rows of any stride and start give the
    same bits, with whole and partial groups of four."""
    from pccl_b200.ops import check_status
    from pccl_b200.ops.gemm import gemm_fp8, quant_blocks, quant_rows
    if stride < K // 128 + shift:
        pytest.skip("rows shorter than their scales")
    a = (_rand((200, K), 95).float() * torch.logspace(-1, 1, K // 128, device="cuda").repeat_interleave(128)).bfloat16()
    aq, a_s = quant_rows(a)
    wq, w_s = quant_blocks(_rand((256, K), 96))
    ref = (aq.view(torch.float8_e4m3fn).double() * a_s.double().repeat_interleave(128, 1)) @ (
        wq.view(torch.float8_e4m3fn).double() * w_s.double().repeat_interleave(128, 0).repeat_interleave(128, 1)).t()
    rows = torch.full((200, stride), float("nan"), device="cuda")
    rows[:, shift:shift + K // 128] = a_s
    out = gemm_fp8(aq, rows[:, shift:shift + K // 128], wq, w_s, out_dtype=torch.float32)
    check_status("gemm_fp8")
    assert torch.equal(out, gemm_fp8(aq, a_s, wq, w_s, out_dtype=torch.float32))
    assert (out.double() - ref).abs().max().item() <= 2e-3 * max(1.0, ref.abs().max().item())


@pytest.mark.parametrize("M,N,K,width", [(12546, 392, 128, 224), (2100, 4360, 640, 192), (18947, 136, 256, 160), (1531, 3584, 1152, 160), (1000, 4096, 256, 128),
                                         (19000, 112, 384, 128), (9490, 232, 1152, 96), (18965, 40, 512, 64)])
def test_mx8_cta_pairs(M, N, K, width):
    """The CTA-pair form at every width the launch picks: ragged rows and columns, tiles that straddle a block of scales, one to nine
    K blocks (a scale image holds four); fp32 and bf16 outputs, bias, GELU and accumulation in the epilogue."""
    from pccl_b200._native import C
    from pccl_b200.ops import check_status
    from pccl_b200.ops.gemm import dequant_rows, gemm_mx8, quant_rows_mx, ue8m0_to_float
    assert C.gemm_mx8_pair_tile_n(M, N, 148) == width
    # magnitudes that differ per K block, per 32 rows and per 128 columns, so that a scale of another place shows
    a = (_rand((M, K), 97).float() * torch.logspace(-1, 1, K // 128, device="cuda").repeat_interleave(128)
         * (1.0 + (torch.arange(M, device="cuda") // 32 % 8).float())[:, None]).bfloat16()
    w = (_rand((N, K), 98, 0.05).float() * (1.0 + (torch.arange(N, device="cuda") // 128 % 5).float())[:, None]).bfloat16()
    aq, a_s = quant_rows_mx(a)
    wq, w_rows = quant_rows_mx(w)
    w_s = w_rows[::128].contiguous()
    ref = dequant_rows(aq, ue8m0_to_float(a_s)).double() @ (
        wq.view(torch.float8_e4m3fn).double() * ue8m0_to_float(w_s).double().repeat_interleave(128, 1).repeat_interleave(128, 0)[:N]).t()
    out = gemm_mx8(aq, a_s, wq, w_s, out_dtype=torch.float32)
    check_status("gemm_mx8 pairs")
    top = max(1.0, ref.abs().max().item())
    assert (out.double() - ref).abs().max().item() <= 2e-3 * top            # sums in another order; a wrong scale or tile is off by O(1)
    bias = _rand((N,), 99)
    old = _rand((M, N), 100)
    got = old.clone()
    gemm_mx8(aq, a_s, wq, w_s, out=got, bias=bias, accumulate=True)
    act = gemm_mx8(aq, a_s, wq, w_s, bias=bias, gelu_inplace=True)
    check_status("gemm_mx8 pairs")
    full = out.double() + bias.double()
    assert ((got.double() - full - old.double()).abs() <= 2 ** -8 * (full + old.double()).abs() + 1e-4).all()
    want = torch.nn.functional.gelu(full, approximate="tanh")
    assert ((act.double() - want).abs() <= 2 ** -8 * want.abs() + 1.5e-3 * full.abs() + 1e-4).all()


@pytest.mark.parametrize("M,N,K", [(1, 8, 64), (17, 200, 72), (128, 512, 256), (129, 264, 64), (130, 200, 136), (777, 3072, 768), (1531, 1000, 264)])
@pytest.mark.parametrize("pair", [None, False, True])
def test_gelu_in_place_is_the_side_output(M, N, K, pair):
    """With ``gelu_inplace`` the output is what ``gelu_out`` gets, bit for bit, whichever kernel the row count picks."""
    from pccl_b200.ops.gemm import check_status, gemm
    torch.manual_seed(M)
    a, b, bias = (torch.randn(*s, device="cuda").bfloat16() for s in ((M, K), (N, K), (N,)))
    act = torch.empty(M, N, device="cuda", dtype=torch.bfloat16)
    gemm(a, b, bias=bias, gelu_out=act, pair=pair)
    assert torch.equal(gemm(a, b, bias=bias, gelu_inplace=True, pair=pair), act)
    check_status()
    with pytest.raises(ValueError):
        gemm(a, b, bias=bias, gelu_out=act, gelu_inplace=True)
