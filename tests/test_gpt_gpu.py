"""The GPT model on this package's kernels against the same network written with stock PyTorch ops
in fp32, and the sharded data-parallel step with a world of one."""
import math

import pytest
import torch
import torch.nn.functional as F

pytestmark = pytest.mark.gpu


def _reference_loss(model, ids, targets):
    """Same weights, fp32 math, stock ops."""
    cfg = model.cfg
    f = lambda t: t.detach().float().requires_grad_(True)  # noqa: E731
    P = {n: f(p) for n, p in model.named_parameters()}
    B, T = ids.shape
    x = P["wte.weight"][ids] + P["wpe.weight"][torch.arange(T, device=ids.device)][None]
    for i in range(cfg.n_layer):
        g = lambda n: P[f"blocks.{i}.{n}"]  # noqa: E731
        h = F.layer_norm(x, (cfg.d_model,), g("ln1.weight"), g("ln1.bias"))
        qkv = F.linear(h, g("qkv.weight"), g("qkv.bias")).view(B, T, 3, cfg.n_head, -1)
        q, k, v = (qkv[:, :, j].transpose(1, 2) for j in range(3))
        a = F.scaled_dot_product_attention(q, k, v, is_causal=True).transpose(1, 2).reshape(B, T, -1)
        x = x + F.linear(a, g("proj.weight"), g("proj.bias"))
        h = F.layer_norm(x, (cfg.d_model,), g("ln2.weight"), g("ln2.bias"))
        x = x + F.linear(F.gelu(F.linear(h, g("fc1.weight"), g("fc1.bias")), approximate="tanh"), g("fc2.weight"), g("fc2.bias"))
    x = F.layer_norm(x, (cfg.d_model,), P["ln_f.weight"], P["ln_f.bias"])
    loss = F.cross_entropy(F.linear(x, P["wte.weight"]).view(B * T, -1), targets.reshape(-1))
    loss.backward()
    return loss.item(), {n: p.grad for n, p in P.items()}


def test_gpt_forward_backward_matches_fp32_reference():
    from pccl_b200.models import GPT, GPTConfig
    from pccl_b200.ops import check_status
    torch.manual_seed(0)
    cfg = GPTConfig.tiny()
    model = GPT(cfg, device="cuda")
    ids = torch.randint(0, cfg.vocab_size, (4, cfg.seq_len), device="cuda")
    tgt = ids.roll(-1, 1)
    loss = model(ids, tgt)
    loss.backward()
    check_status("gpt")
    ref_loss, ref_grads = _reference_loss(model, ids, tgt)
    assert abs(loss.item() - ref_loss) < 0.02 * ref_loss
    for name in ("blocks.0.qkv.weight", "blocks.1.fc1.weight", "blocks.1.fc2.weight", "blocks.0.proj.bias", "wte.weight",
                 "wpe.weight", "blocks.1.ln2.weight", "blocks.0.fc1.bias", "blocks.1.fc2.bias", "blocks.0.fc2.bias", "blocks.1.qkv.bias",
                 "blocks.0.ln1.weight", "ln_f.bias"):
        got = dict(model.named_parameters())[name].grad.float()
        ref = ref_grads[name]
        denom = ref.abs().max().item() + 1e-8
        assert (got - ref).abs().max().item() / denom < 0.08, name


def test_fused_cross_entropy_matches_torch():
    from pccl_b200.nn import fused_cross_entropy
    torch.manual_seed(1)
    rows, vocab, ld = 300, 50257, 50264
    store = (torch.randn(rows, ld, device="cuda") * 3).bfloat16()
    logits = store[:, :vocab]
    tgt = torch.randint(0, vocab, (rows,), device="cuda")
    ref_in = logits.float().clone().requires_grad_(True)
    ref = F.cross_entropy(ref_in, tgt)
    ref.backward()
    x = logits.clone().as_strided(logits.shape, logits.stride()) if False else store.clone()[:, :vocab]
    x.requires_grad_(True)
    loss = fused_cross_entropy(x, tgt)
    loss.backward()
    assert abs(loss.item() - ref.item()) < 1e-3
    assert (x.grad.float() - ref_in.grad).abs().max().item() < 2e-5 + 0.01 * ref_in.grad.abs().max().item()


def test_cross_entropy_reports_a_target_outside_the_vocabulary_instead_of_indexing_with_it():
    """An out-of-range target is never used as an index: its row gets loss 0 and a zero gradient, the first such
    row is written to the device status words, and ``ignore_index`` itself stays silent."""
    from pccl_b200.ops import check_status
    from pccl_b200.ops.elementwise import cross_entropy_
    import pytest as _pt
    torch.manual_seed(5)
    rows, vocab = 32, 512
    x = (torch.randn(rows, vocab, device="cuda") * 2).bfloat16()
    tgt = torch.randint(0, vocab, (rows,), device="cuda")
    tgt[5] = -100
    check_status("before")
    quiet = cross_entropy_(x.clone(), tgt, grad_scale=1.0, ignore_index=-100)
    check_status("ignore_index is not an error")
    assert quiet[5].item() == 0.0
    tgt[9] = vocab + 3
    y = x.clone()
    loss = cross_entropy_(y, tgt, grad_scale=1.0, ignore_index=-100)
    assert loss[9].item() == 0.0 and int(y[9].abs().sum()) == 0 and loss[8].item() > 0.0
    with _pt.raises(RuntimeError, match="device status"):
        check_status("cross entropy with a bad target")
    check_status("cleared")


def test_adamw_kernel_matches_torch():
    from pccl_b200.ops.elementwise import adamw_step
    torch.manual_seed(2)
    n = 100003
    p = torch.randn(n, device="cuda"); g = torch.randn(n, device="cuda") * 0.1
    ref_p = p.clone().requires_grad_(True)
    opt = torch.optim.AdamW([ref_p], lr=1e-2, betas=(0.9, 0.95), eps=1e-8, weight_decay=0.1)
    m, v, out = torch.zeros_like(p), torch.zeros_like(p), torch.empty(n, device="cuda", dtype=torch.bfloat16)
    for step in (1, 2, 3):
        ref_p.grad = g.clone() * step
        opt.step()
        adamw_step(p, m, v, g * step, out, lr=1e-2, betas=(0.9, 0.95), eps=1e-8, weight_decay=0.1, step=step)
    assert (p - ref_p.detach()).abs().max().item() < 1e-5
    assert torch.equal(out, p.bfloat16())


@pytest.mark.parametrize("n", [8, 504, 520, 2048, 2056, 303112, 1212424, (32 << 20) + 24])
@pytest.mark.parametrize("beside", [False, True])
def test_bucket_update_in_a_world_of_one(n, beside):
    """Whole and partial trips of a warp, more trips than CTAs, one launch and several, and the size from which more CTAs run; two steps against the formula in
    fp64 (each step rounds master and moments to fp32 a few times: 1e-5), parameters one bf16 rounding of the masters."""
    import torch
    from pccl_b200.engine import Engine
    from pccl_b200.ops import collectives as coll
    torch.manual_seed(n % 1000)
    eng = Engine(0, 1)
    eng.initEngine("cuda", 2 * n + (640 << 20))
    g = eng.symmetric_tensor((n,), torch.bfloat16, align=256)
    pad = torch.full((n + 64,), 7.0, dtype=torch.bfloat16, device="cuda")
    out = pad[32:32 + n]
    p, m, v = torch.randn(n, device="cuda"), torch.zeros(n, device="cuda"), torch.zeros(n, device="cuda")
    p64, m64, v64 = p.double(), m.double(), v.double()
    for step in (1, 2):
        g.copy_(torch.randn(n, device="cuda"))
        coll.reduce_scatter_adamw(eng, g, p, m, v, out, lr=1e-2, betas=(0.9, 0.95), eps=1e-8, weight_decay=0.1, step=step, scale=0.5, beside=beside)
        g64 = g.double() * 0.5
        m64, v64 = 0.9 * m64 + 0.1 * g64, 0.95 * v64 + 0.05 * g64 * g64
        p64 = p64 * (1 - 1e-2 * 0.1) - 1e-2 * (m64 / (1 - 0.9 ** step)) / ((v64 / (1 - 0.95 ** step)).sqrt() + 1e-8)
    for got, want in ((p, p64), (m, m64), (v, v64)):
        assert (got.double() - want).abs().max().item() <= 1e-5 * max(1.0, want.abs().max().item())
    assert torch.equal(out, p.bfloat16())
    assert (pad[:32] == 7).all() and (pad[32 + n:] == 7).all()


def test_launches_of_the_bucket_update_are_counted():
    from pccl_b200.engine import Engine
    from pccl_b200.ops import collectives as coll, launch_count
    n = 303112
    eng = Engine(0, 1)
    eng.initEngine("cuda", 640 << 20)
    g = eng.symmetric_tensor((n,), torch.bfloat16, align=256)
    g.zero_()
    p, m, v = (torch.zeros(n, device="cuda") for _ in range(3))
    out = torch.empty(n, device="cuda", dtype=torch.bfloat16)
    for blocks, threads, launches in ((None, 512, 1), (1, 128, 38), (2, 128, 19)):        # 8192 parameters per CTA of 128 threads and launch; 148 CTAs
        before = launch_count()
        coll.reduce_scatter_adamw(eng, g, p, m, v, out, lr=1e-2, blocks=blocks, threads=threads, beside=True)
        assert launch_count() - before == launches
    torch.cuda.synchronize()


def test_bucket_update_with_a_block_count_of_the_callers(monkeypatch):
    """A wrapper hands its own count on, none otherwise; any count gives the same bits."""
    from pccl_b200.models import GPT, GPTConfig
    from pccl_b200.ops import collectives as coll
    from pccl_b200.parallel.dp import ShardedDataParallel
    seen, update = [], coll.reduce_scatter_adamw
    monkeypatch.setattr(coll, "reduce_scatter_adamw", lambda *a, **k: (seen.append(k["blocks"]), update(*a, **k)))
    masters = []
    for blocks in (None, 3):
        torch.manual_seed(1)
        model = GPT(GPTConfig.tiny(), device="cuda")
        dp = ShardedDataParallel(model, heap_bytes=256 << 20, comm_blocks=blocks)
        seen.clear()
        dp.zero_grad()
        for b in dp.buckets:                                   # the update alone: gradients made here
            b.grads.copy_(torch.randn(b.numel, device="cuda"))
            dp._launch_reduce(b)
        torch.cuda.synchronize()
        assert seen and set(seen) == {blocks}
        masters.append([b.master.clone() for b in dp.buckets])
    assert all(torch.equal(a, b) for a, b in zip(*masters))


@pytest.mark.parametrize("fused", [True, False])
def test_stream_priority_in_a_world_of_one(fused):
    """The plain reduce-scatter and optimizer of the unfused mode go first; the fused update's short launches do not."""
    from pccl_b200.models import GPT, GPTConfig
    from pccl_b200.parallel.dp import ShardedDataParallel
    torch.manual_seed(1)
    dp = ShardedDataParallel(GPT(GPTConfig.tiny(), device="cuda"), heap_bytes=256 << 20, fuse_optimizer=fused)
    assert dp.comm_stream.priority == (0 if fused else -1)
    ids = torch.randint(0, 1001, (2, 128), device="cuda")
    losses = [dp.train_step(ids, ids.roll(-1, 1)).item() for _ in range(3)]
    assert losses[-1] < losses[0]


def test_sharded_dp_world_of_one_trains_and_matches_plain_adamw():
    from pccl_b200.models import GPT, GPTConfig
    from pccl_b200.models.gpt import smoke_step
    from pccl_b200.ops import check_status, launch_count
    before = launch_count()
    last = smoke_step()
    check_status("dp")
    assert math.isfinite(last) and launch_count() - before > 50


def test_fused_and_unfused_optimizer_paths_agree():
    """Reduce-scatter + AdamW in one kernel gives the parameters of the two-kernel path."""
    from pccl_b200.engine import Engine
    from pccl_b200.models import GPT, GPTConfig
    from pccl_b200.parallel import ShardedDataParallel
    cfg = GPTConfig.tiny()
    ids = torch.randint(0, cfg.vocab_size, (2, cfg.seq_len), device="cuda", generator=torch.Generator(device="cuda").manual_seed(3))
    flats = []
    for fused in (True, False):
        torch.manual_seed(0)
        model = GPT(cfg, device="cuda")
        eng = Engine(0, 1); eng.initEngine("cuda", heap_bytes=256 << 20)
        dp = ShardedDataParallel(model, eng, lr=1e-3, bucket_mb=0.5, fuse_optimizer=fused)
        for _ in range(2):
            dp.train_step(ids, ids.roll(-1, 1))
        torch.cuda.synchronize()
        flats.append(dp.flat_params.float().clone())
        del dp, model, eng
    assert (flats[0] - flats[1]).abs().max().item() <= 2e-2 * flats[1].abs().max().item()
    assert (flats[0] == flats[1]).float().mean().item() > 0.9       # identical except where atomics order / bf16 rounding of a gradient differs


def test_an_untied_head_above_32_mi_parameters_is_updated_while_backward_runs():
    """Its bucket is the first to complete and goes out as one wide launch: the same parameters as with the optimizer behind the backward pass."""
    from pccl_b200.models import GPT, GPTConfig
    from pccl_b200.parallel import ShardedDataParallel
    cfg = GPTConfig(n_layer=1, n_head=16, d_model=2048, seq_len=64, vocab_size=16401, tie_embeddings=False)
    ids = torch.randint(0, cfg.vocab_size, (2, 64), device="cuda", generator=torch.Generator(device="cuda").manual_seed(3))
    got = []
    for fused in (True, False):
        torch.manual_seed(0)
        dp = ShardedDataParallel(GPT(cfg, device="cuda"), lr=1e-3, fuse_optimizer=fused)
        assert dp.buckets[0].numel > 32 << 20 and dp.buckets[0].params[0] is dp.model.lm_head.weight
        dp.train_step(ids, ids.roll(-1, 1))
        torch.cuda.synchronize()
        got.append({n: p.detach().clone() for n, p in dp.model.named_parameters()})
    for name, p in got[0].items():
        if name == "wte.weight":                               # its gradient is a sum in no fixed order
            assert (p == got[1][name]).float().mean().item() > 0.99
        else:
            assert torch.equal(p, got[1][name]), name


def test_timed_step_reports_every_bucket_and_trains_like_train_step():
    """The opt-in per-bucket timing takes the same step as train_step and returns ordered, non-negative spans."""
    from pccl_b200.engine import Engine
    from pccl_b200.models import GPT, GPTConfig
    from pccl_b200.parallel import ShardedDataParallel
    cfg = GPTConfig.tiny()
    ids = torch.randint(0, cfg.vocab_size, (2, cfg.seq_len), device="cuda", generator=torch.Generator(device="cuda").manual_seed(3))
    flats = []
    for timed in (False, True):
        torch.manual_seed(0)
        model = GPT(cfg, device="cuda")
        eng = Engine(0, 1); eng.initEngine("cuda", heap_bytes=256 << 20)
        dp = ShardedDataParallel(model, eng, lr=1e-3, bucket_mb=0.5)
        dp.train_step(ids, ids.roll(-1, 1))
        if timed:
            rep = dp.timed_step(ids, ids.roll(-1, 1))
            assert len(rep["buckets"]) == len(dp.buckets) and math.isfinite(rep["loss"])
            assert 0 < rep["forward_end"] < rep["backward_end"] <= rep["step_end"]
            for row in rep["buckets"]:
                assert row["ready"] <= row["start"] + 1e-3 and row["start"] <= row["reduced"] <= row["done"] <= rep["step_end"] + 1e-3
            assert rep["exposed_ms"] >= 0 and rep["comm_busy_ms"] > 0
        else:
            dp.train_step(ids, ids.roll(-1, 1))
        torch.cuda.synchronize()
        flats.append(dp.flat_params.float().clone())
        del dp, model, eng
    assert (flats[0] - flats[1]).abs().max().item() <= 2e-2 * flats[1].abs().max().item()


def test_dp_checkpoint_resume_matches_uninterrupted_training(tmp_path):
    """torch.save of the sharded optimizer state and flat parameters after two steps, loaded into a differently
    initialised trainer, continues like the run that was never interrupted."""
    from pccl_b200.engine import Engine
    from pccl_b200.models import GPT, GPTConfig
    from pccl_b200.parallel import ShardedDataParallel
    cfg = GPTConfig.tiny()
    ids = torch.randint(0, cfg.vocab_size, (2, cfg.seq_len), device="cuda", generator=torch.Generator(device="cuda").manual_seed(5))

    def make(seed):
        torch.manual_seed(seed)
        model = GPT(cfg, device="cuda")
        eng = Engine(0, 1); eng.initEngine("cuda", heap_bytes=256 << 20)
        return model, eng, ShardedDataParallel(model, eng, lr=1e-3, bucket_mb=0.5)

    model, eng, dp = make(0)
    for _ in range(2):
        dp.train_step(ids, ids.roll(-1, 1))
    torch.cuda.synchronize()
    torch.save(dp.gather_full_state(), tmp_path / "ckpt.pt")
    for _ in range(2):
        last = float(dp.train_step(ids, ids.roll(-1, 1)))
    torch.cuda.synchronize()
    want = dp.flat_params.float().clone()
    del dp, model, eng
    model, eng, dp = make(1)            # other initial weights: everything has to come from the checkpoint
    dp.load_full_state(torch.load(tmp_path / "ckpt.pt"))
    assert dp.step_count == 2
    for _ in range(2):
        resumed = float(dp.train_step(ids, ids.roll(-1, 1)))
    torch.cuda.synchronize()
    got = dp.flat_params.float()
    assert abs(resumed - last) <= 2e-2 * abs(last), (resumed, last)
    assert (got - want).abs().max().item() <= 2e-2 * want.abs().max().item()
    assert (got == want).float().mean().item() > 0.9


@pytest.mark.parametrize("rows,D", [(37, 256), (4096, 2048), (600, 4096), (130, 8192)])
def test_layernorm_kernels_match_fp32_reference(rows, D):
    from pccl_b200.nn import LayerNorm
    torch.manual_seed(5)
    ln = LayerNorm(D, device="cuda")
    with torch.no_grad():
        ln.weight.copy_((torch.randn(D, device="cuda") * 0.5 + 1).bfloat16())
        ln.bias.copy_((torch.randn(D, device="cuda") * 0.1).bfloat16())
    x = (torch.randn(rows, D, device="cuda") * 2 + 0.5).bfloat16().requires_grad_(True)
    g = torch.randn(rows, D, device="cuda").bfloat16()
    y = ln(x)
    y.backward(g)
    xr = x.detach().float().requires_grad_(True)
    wr = ln.weight.detach().float().requires_grad_(True)
    br = ln.bias.detach().float().requires_grad_(True)
    yr = F.layer_norm(xr, (D,), wr, br, 1e-5)
    yr.backward(g.float())
    assert ((y.float() - yr).abs() <= 0.01 + 0.008 * yr.abs()).all()       # one bf16 rounding of the output
    assert (x.grad.float() - xr.grad).abs().max().item() < 0.03 * max(1.0, xr.grad.abs().max().item())
    assert (ln.weight.grad.float() - wr.grad).abs().max().item() < 0.02 * max(1.0, wr.grad.abs().max().item())
    assert (ln.bias.grad.float() - br.grad).abs().max().item() < 0.02 * max(1.0, br.grad.abs().max().item())


@pytest.mark.parametrize("rows,D", [(512, 2048), (300, 256), (64, 4096)])
def test_fused_residual_add_layernorm_matches_fp32_reference(rows, D):
    """(x, delta) -> (x + delta, LN(x + delta)) forward, and backward with the gradient on the residual stream added in
    and the producing layer's bias gradient (column sums of d delta) as a by-product."""
    from pccl_b200.nn import LayerNorm
    torch.manual_seed(7)
    ln = LayerNorm(D, device="cuda")
    with torch.no_grad():
        ln.weight.copy_((1 + 0.1 * torch.randn(D, device="cuda")).bfloat16())
        ln.bias.copy_((0.1 * torch.randn(D, device="cuda")).bfloat16())
    x = torch.randn(rows, D, device="cuda").bfloat16().requires_grad_(True)
    delta = torch.randn(rows, D, device="cuda").bfloat16().requires_grad_(True)
    prev_bias = torch.zeros(D, device="cuda", dtype=torch.bfloat16, requires_grad=True)
    s, y = ln.add_norm(x, delta, prev_bias)
    gs, gy = torch.randn(rows, D, device="cuda").bfloat16(), torch.randn(rows, D, device="cuda").bfloat16()
    torch.autograd.backward([s, y], [gs, gy])
    xr, dr = x.detach().float().requires_grad_(True), delta.detach().float().requires_grad_(True)
    wr, br = ln.weight.detach().float().requires_grad_(True), ln.bias.detach().float().requires_grad_(True)
    # the norm sees the stored (bf16-rounded) sum; gradients pass straight through the rounding
    sr = (xr + dr) + ((xr + dr).detach().bfloat16().float() - (xr + dr).detach())
    yr = F.layer_norm(sr, (D,), wr, br, ln.eps)
    torch.autograd.backward([sr, yr], [gs.float(), gy.float()])
    assert (s.float() - sr).abs().max().item() <= 1e-6
    assert (y.float() - yr).abs().max().item() <= 3e-2
    tol = 3e-2 * max(1.0, xr.grad.abs().max().item())
    assert (x.grad.float() - xr.grad).abs().max().item() <= tol
    assert x.grad.data_ptr() == delta.grad.data_ptr() or torch.equal(x.grad, delta.grad)
    for got, ref in ((ln.weight.grad, wr.grad), (ln.bias.grad, br.grad), (prev_bias.grad, dr.grad.sum(0))):
        assert (got.float() - ref).abs().max().item() <= 2e-2 * max(1.0, ref.abs().max().item())


# edges of the rules that pick the forward kernel's form (148 SMs): one row per CTA up to one row per SM and from three on, the widths at which a
# thread takes another vector, 6 and 8 rows per SM with eight warps, 4 and 7 Mi values
@pytest.mark.parametrize("rows,D", [(148, 264), (149, 1032), (444, 1032), (445, 1032), (2048, 2048), (2049, 2048), (3, 2056), (445, 2056), (889, 4096), (1185, 4096),
                                    (2389, 3072), (2390, 3072), (5, 4104), (445, 5120), (448, 5128), (148, 6152), (149, 8192), (445, 8192)])
def test_layernorm_forward_at_the_edges_of_its_forms(rows, D):
    from pccl_b200.nn.norm import _ln_forward
    torch.manual_seed(rows + D)
    x, delta = (torch.randn(rows, D, device="cuda") * 2 + 0.5).bfloat16(), torch.randn(rows, D, device="cuda").bfloat16()
    w, b = (torch.randn(D, device="cuda") * 0.5 + 1).bfloat16(), torch.randn(D, device="cuda").bfloat16()
    for d in (None, delta):
        s, y, stats = _ln_forward(x, d, w, b, 1e-5)
        base = x if d is None else (x.float() + d.float()).bfloat16()      # the norm sees the sum as it is stored
        assert d is None or torch.equal(s, base)
        ref = F.layer_norm(base.double(), (D,), w.double(), b.double(), 1e-5)
        # a bf16 result is rounded by half of 2^-8; fp32 sums of up to 8192 terms and rsqrt leave some 1e-6 of a normalised value (at most 6 here) times w
        assert ((y.double() - ref).abs() <= 2 ** -8 * ref.abs() + 1e-4).all()
        assert (stats[0].double() - base.double().mean(1)).abs().max().item() < 1e-5
        rstd = (base.double().var(1, unbiased=False) + 1e-5).rsqrt()
        assert (stats[1].double() / rstd - 1).abs().max().item() < 1e-5


# edges of the rule for the ring (7 and 16 rows per SM) and of the widths at which the kernel changes
@pytest.mark.parametrize("rows,D", [(1, 2056), (3, 4096), (2368, 2056), (2369, 2056), (300, 3080), (1, 8192), (1036, 4104), (1037, 4104), (149, 6152)])
def test_layernorm_backward_with_and_without_its_ring(rows, D):
    from pccl_b200.nn.norm import _ln_backward, _ln_forward
    torch.manual_seed(rows + D)
    x, dy, dres = (torch.randn(rows, D, device="cuda").bfloat16() for _ in range(3))
    w, b = (torch.randn(D, device="cuda") * 0.5 + 1).bfloat16(), torch.zeros(D, device="cuda", dtype=torch.bfloat16)
    stats = _ln_forward(x, None, w, b, 1e-5)[2]
    dg, db, dc = (torch.empty_like(w) for _ in range(3))
    dx = _ln_backward(dy, x, w, stats, dres, dg, db, dc).double()
    xd, g = x.double(), dy.double() * w.double()
    xh = (xd - xd.mean(1, keepdim=True)) * (xd.var(1, unbiased=False, keepdim=True) + 1e-5).rsqrt()
    rs = (xd.var(1, unbiased=False, keepdim=True) + 1e-5).rsqrt()
    ref = rs * (g - g.mean(1, keepdim=True) - xh * (g * xh).mean(1, keepdim=True)) + dres.double()
    assert ((dx - ref).abs() <= 2 ** -8 * ref.abs() + 1e-4).all()              # the rounding of bf16, and fp32 arithmetic on values of some 20
    # column sums in fp32, rounded to bf16: 2^-8 of the sum and some 1e-6 of the terms' sizes
    for got, terms in ((dg, dy.double() * xh), (db, dy.double()), (dc, ref)):
        assert ((got.double() - terms.sum(0)).abs() <= 2 ** -8 * terms.sum(0).abs() + 1e-5 * terms.abs().sum(0) + 1e-6).all()


def test_fused_mlp_backward_matches_fp32_reference():
    """fc2(gelu(fc1(x))) as one autograd node (GELU derivative and first bias gradient inside the GEMM epilogue)."""
    from pccl_b200.nn import Linear, mlp
    torch.manual_seed(8)
    rows, d, h = 512, 256, 1024
    fc1, fc2 = Linear(d, h, device="cuda"), Linear(h, d, device="cuda")
    with torch.no_grad():
        fc1.bias.copy_((0.1 * torch.randn(h, device="cuda")).bfloat16())
        fc2.bias.copy_((0.1 * torch.randn(d, device="cuda")).bfloat16())
    x = torch.randn(rows, d, device="cuda").bfloat16().requires_grad_(True)
    g = torch.randn(rows, d, device="cuda").bfloat16()
    mlp(x, fc1, fc2).backward(g)
    xr = x.detach().float().requires_grad_(True)
    P = {n: p.detach().float().requires_grad_(True) for n, p in (("w1", fc1.weight), ("b1", fc1.bias), ("w2", fc2.weight), ("b2", fc2.bias))}
    out = F.linear(F.gelu(F.linear(xr, P["w1"], P["b1"]), approximate="tanh"), P["w2"], P["b2"])
    out.backward(g.float())
    for got, ref, name in ((x.grad, xr.grad, "dx"), (fc1.weight.grad, P["w1"].grad, "dw1"), (fc1.bias.grad, P["b1"].grad, "db1"),
                           (fc2.weight.grad, P["w2"].grad, "dw2"), (fc2.bias.grad, P["b2"].grad, "db2")):
        assert (got.float() - ref).abs().max().item() <= 5e-2 * max(1e-3, ref.abs().max().item()), name
    # the second bias gradient can be left to the consumer of the output
    fc2.bias.grad = None
    mlp(x, fc1, fc2, defer_fc2_bias_grad=True).backward(g)
    assert fc2.bias.grad is None


def test_norm_gradients_reach_the_buckets_by_either_way():
    """A norm used once is written into the flat bucket by the kernel; one that is used twice, or whose weight has a hook,
    travels through autograd.  Both end in the gradient that plain autograd gives (bf16 sums of two terms: 2^-7)."""
    import torch
    import torch.nn as nn
    from pccl_b200.nn import LayerNorm, Linear
    from pccl_b200.parallel.dp import ShardedDataParallel

    class Net(nn.Module):
        def __init__(self):
            super().__init__()
            self.once, self.twice, self.hooked = (LayerNorm(64, device="cuda") for _ in range(3))
            self.lin = Linear(64, 64, device="cuda", init_std=0.3)

        def forward(self, x, t):
            h = self.twice(self.lin(self.once(x)))
            return (self.hooked(self.twice(h + x)) * t).float().mean()

    torch.manual_seed(3)
    net = Net()
    x, t = torch.randn(40, 64, device="cuda").bfloat16(), torch.randn(40, 64, device="cuda").bfloat16()
    ref = torch.autograd.grad(net(x, t), list(net.parameters()))
    seen = []
    net.hooked.weight.register_hook(lambda g: seen.append(g.shape))
    dp = ShardedDataParallel(net, heap_bytes=64 << 20)
    for step in range(2):
        dp.zero_grad()
        net(x, t).backward()
        if step == 0:                                     # before the update changes the parameters
            for p, g in zip(net.parameters(), ref):
                assert (p.main_grad.float() - g.float()).abs().max().item() <= 2 ** -7 * g.float().abs().max().item() + 1e-6
        dp.optimizer_step()
    assert len(seen) == 2 and all(p.grad is None for p in net.parameters())


def test_forward_without_gradients_is_the_same_forward():
    """Without gradients the layers run outside autograd.Function: same kernels, same bits, and transforms still refuse."""
    import torch
    from pccl_b200.nn import LayerNorm, Linear, LinearGelu, mlp
    torch.manual_seed(4)
    x, d = (torch.randn(3, 50, 72, device="cuda").bfloat16() for _ in range(2))
    fc1, fc2, ln = LinearGelu(72, 96, device="cuda"), Linear(96, 72, device="cuda"), LayerNorm(72, device="cuda")
    calls = [lambda: fc2(fc1(x), residual=d), lambda: mlp(x, fc1, fc2), lambda: ln(x), lambda: ln.add_norm(x, d)[0], lambda: ln.add_norm(x, d)[1]]
    for f in calls:
        with torch.no_grad():
            plain = f()
        assert torch.equal(plain, f().detach())
    with torch.no_grad(), pytest.raises(RuntimeError):
        torch.vmap(lambda v: ln(v))(x)


@pytest.mark.parametrize("D", [8, 64, 256, 264, 768, 1544, 2048, 2056, 4096, 8192])
@pytest.mark.parametrize("rows", [1, 5, 700, 5003])
def test_layer_norm_backward_over_widths(D, rows):
    """With and without the residual gradient and the column sums of dx.  One to eight warps per row, one to eight rows side by side
    in a CTA, widths off the vector counts, fewer rows than a trip takes and several trips; against fp64 on the same bf16 inputs.  dx is rounded once (2^-8 of its terms), column sums are fp32 sums of `rows`
    terms rounded once."""
    import torch
    from pccl_b200.nn import LayerNorm
    torch.manual_seed(D + rows)
    ln = LayerNorm(D, device="cuda")
    ln.weight.data.copy_(torch.randn(D, device="cuda").bfloat16())
    x, d, gs, gy = (torch.randn(rows, D, device="cuda").bfloat16() for _ in range(4))
    xr, dr = x.clone().requires_grad_(True), d.clone().requires_grad_(True)
    prev = torch.nn.Parameter(torch.zeros(D, device="cuda").bfloat16())
    s, y = ln.add_norm(xr, dr, prev)
    got = torch.autograd.grad([s, y], [xr, ln.weight, ln.bias, prev], [gs, gy])
    s64 = s.detach().double().requires_grad_(True)
    w64, b64 = ln.weight.detach().double().requires_grad_(True), torch.zeros(D, device="cuda", dtype=torch.float64, requires_grad=True)
    y64 = F.layer_norm(s64, (D,), w64, b64, ln.eps)
    dx, dw, db = torch.autograd.grad(y64, [s64, w64, b64], gy.double())
    sr = s.detach().requires_grad_(True)
    plain = torch.autograd.grad(ln(sr), [sr, ln.weight, ln.bias], gy)
    for a, b in zip(plain, (dx, dw, db)):
        assert (a.double() - b).abs().max().item() <= 2 ** -8 * b.abs().max().item() + 1e-4
    dx = dx + gs.double()
    for a, b in zip(got, (dx, dw, db, dx.sum(0))):
        assert (a.double() - b).abs().max().item() <= 2 ** -8 * b.abs().max().item() + 1e-4


@pytest.mark.parametrize("D", [8, 248, 264, 512, 520, 776, 1024, 1032, 2048, 2056, 4104, 8192])
@pytest.mark.parametrize("rows", [1, 297, 5003, 17001])
def test_layer_norm_forward_over_widths(D, rows):
    """One to eight warps per row with one to four vectors per thread, rows that do not fill the last CTA, and the row counts at which
    the launch goes from one vector per thread to as many as fit.  Against fp64 on the same bf16 inputs: the sum is rounded to bf16
    once and compared exactly, the statistics are fp32 sums (1e-5), the result is rounded once."""
    import torch
    from pccl_b200.nn.norm import _ln_forward
    torch.manual_seed(D + rows)
    x, d = ((torch.randn(rows, D, device="cuda") + 3.0).bfloat16() for _ in range(2))
    w, b = (torch.randn(D, device="cuda").bfloat16() for _ in range(2))
    for delta in (None, d):
        s, y, stats = _ln_forward(x, delta, w, b, 1e-5)
        total = x if delta is None else (x.float() + d.float()).bfloat16()
        assert s is None or torch.equal(s, total)
        t = total.double()
        var = t.var(1, unbiased=False)
        assert torch.allclose(stats[0].double(), t.mean(1), rtol=1e-5, atol=1e-6)
        assert torch.allclose(stats[1].double(), (var + 1e-5).rsqrt(), rtol=1e-4)
        ref = F.layer_norm(t, (D,), w.double(), b.double(), 1e-5)
        assert ((y.double() - ref).abs() <= 2 ** -8 * ref.abs() + 1e-4 * (1 + ref.abs().max())).all()


@pytest.mark.parametrize("vocab", [7, 1001, 50257])
def test_cross_entropy_with_masked_and_large_logits(vocab):
    """Logits of -inf (masked classes, whole stretches of them), of the type's lowest value and of +-3e4: the running maximum starts
    at -inf and grows late in the row."""
    import torch
    from pccl_b200.ops.elementwise import cross_entropy_
    torch.manual_seed(vocab)
    ld = (vocab + 7) // 8 * 8
    lg = (torch.randn(6, ld, device="cuda") * 4).bfloat16()[:, :vocab]
    lg[1, : vocab // 2] = float("-inf")
    lg[2, vocab // 2:] = float("-inf")
    lg[3] = torch.finfo(torch.bfloat16).min
    lg[4] = torch.linspace(-3e4, 3e4, vocab, device="cuda").bfloat16()
    lg[5, : vocab - 1] = float("-inf")
    tgt = torch.tensor([0, vocab - 1, 0, 3, vocab - 1, vocab - 1], device="cuda")
    ref = lg.double().requires_grad_(True)
    loss64 = F.cross_entropy(ref, tgt, reduction="none")
    g64, = torch.autograd.grad(loss64.sum(), ref)
    loss = cross_entropy_(lg, tgt)
    assert ((loss.double() - loss64).abs() <= 1e-5 * loss64.abs() + 1e-5).all()      # 3e4 in fp32: 2^-24 relative, a few roundings
    assert (lg.double() - g64).abs().max().item() <= 2 ** -8


@pytest.mark.parametrize("B,T,heads,hd", [(1, 1, 1, 8), (2, 77, 3, 24), (3, 130, 2, 64), (1, 300, 5, 128)])
@pytest.mark.parametrize("layout", ["bthd", "bhtd", "odd"])
def test_split_qkv_packs_gradients_and_sums_columns(B, T, heads, hd, layout):
    """Gradients in the layouts that attention kernels return, and one (head dimension not innermost) that is copied first; the
    packed gradient is a copy (exact), its column sums fp32 sums of bf16 values rounded once."""
    import torch
    from pccl_b200.nn.linear import split_qkv
    torch.manual_seed(T)
    qkv = torch.randn(B, T, 3 * heads * hd, device="cuda").bfloat16().requires_grad_(True)
    bias = torch.nn.Parameter(torch.zeros(3 * heads * hd, device="cuda").bfloat16())
    q, k, v = split_qkv(qkv, heads, bias)
    ref = qkv.detach().view(B, T, 3, heads, hd)
    for i, t in enumerate((q, k, v)):
        assert torch.equal(t, ref[:, :, i].transpose(1, 2))
    gs = [torch.randn(B, heads, T, hd, device="cuda").bfloat16() for _ in range(3)]
    if layout == "bthd":
        gs = [g.transpose(1, 2).contiguous().transpose(1, 2) for g in gs]
    elif layout == "odd":
        gs = [g.transpose(2, 3).contiguous().transpose(2, 3) for g in gs]
    dq, db = torch.autograd.grad([q, k, v], [qkv, bias], gs)
    want = torch.stack([g.transpose(1, 2) for g in gs], 2).reshape(B, T, -1)
    assert torch.equal(dq, want)
    sums = want.double().sum((0, 1))
    assert ((db.double() - sums).abs() <= 2 ** -8 * sums.abs() + 1e-4).all()


def _wrapped_norms():
    """x -> norm -> norm under the data-parallel wrapper, inputs, and the gradients that plain autograd gives."""
    import torch.nn as nn
    from pccl_b200.nn import LayerNorm
    from pccl_b200.parallel.dp import ShardedDataParallel

    class Net(nn.Module):
        def __init__(self):
            super().__init__()
            self.a, self.b = (LayerNorm(64, device="cuda") for _ in range(2))

        def forward(self, x, t):
            return (self.b(self.a(x)) * t).float().mean()

    torch.manual_seed(9)
    net = Net()
    for p in net.parameters():
        p.data.add_(torch.randn(64, device="cuda").bfloat16() * 0.3)
    x, t = (torch.randn(40, 64, device="cuda").bfloat16() for _ in range(2))
    x.requires_grad_(True)
    ref = torch.autograd.grad(net(x, t), [x] + list(net.parameters()))
    dp = ShardedDataParallel(net, heap_bytes=64 << 20)
    dp.zero_grad()
    return net, dp, x, t, ref


def test_frozen_norm_is_not_trained():
    net, dp, x, t, _ = _wrapped_norms()
    net.a.weight.requires_grad_(False)
    before = [p.detach().clone() for p in net.parameters()]
    net(x, t).backward()
    assert not net.a.weight._pccl_written and dp.buckets[0].pending == 1
    with pytest.raises(RuntimeError, match="never arrived"):
        dp.optimizer_step()
    torch.cuda.synchronize()
    assert all(torch.equal(p, q) for p, q in zip(net.parameters(), before))


def test_autograd_grad_over_a_wrapped_norm():
    """``autograd.grad`` returns the gradients (in memory of their own) and leaves buckets and their counters alone; the step
    that follows is as if it had not been."""
    net, dp, x, t, ref = _wrapped_norms()
    params = list(net.parameters())
    got = torch.autograd.grad(net(x, t), [x] + params)
    alone, = torch.autograd.grad(net(x, t), [x])
    assert all(torch.equal(a, b) for a, b in zip(got, ref)) and torch.equal(alone, ref[0])
    assert dp.buckets[0].pending == 4 and not dp.flat_grads.any() and not any(p._pccl_written for p in params)
    net(x, t).backward()
    assert all(torch.equal(p.main_grad, g) for p, g in zip(params, ref[1:])) and dp.buckets[0].pending == 0
    dp.optimizer_step()
    assert all(torch.equal(a, b) for a, b in zip(got, ref))


def test_norm_weight_that_the_loss_uses_once_more():
    """A penalty on a norm's weight: the bucket gets the sum of both contributions, once."""
    net, dp, x, t, ref = _wrapped_norms()
    w = net.a.weight.detach().clone()
    (net(x, t) + net.a.weight.float().pow(2).sum()).backward()
    assert [p._pccl_seen for p in net.parameters()] == [1, 1, 1, 1]
    want = ref[1].float() + 2 * w.float()
    assert (net.a.weight.main_grad.float() - want).abs().max().item() <= 2 ** -7 * want.abs().max().item()      # two bf16 terms
    assert all(torch.equal(p.main_grad, g) for p, g in zip(list(net.parameters())[1:], ref[2:]))


def test_gradients_that_hooks_keep_are_not_the_bucket():
    net, dp, x, t, ref = _wrapped_norms()
    kept = []
    net.a.weight.register_hook(kept.append)
    net.b.bias.register_post_accumulate_grad_hook(lambda p: None)
    net(x, t).backward()
    dp.optimizer_step()
    dp.zero_grad()
    (net(x, t) * 3).backward()
    torch.cuda.synchronize()
    assert torch.equal(kept[0], ref[1]) and not torch.equal(kept[1], ref[1])
    assert kept[0].data_ptr() != net.a.weight.main_grad.data_ptr()


def test_norm_bias_may_change_between_forward_and_backward():
    from pccl_b200.nn import LayerNorm
    ln = LayerNorm(64, device="cuda")
    x = torch.randn(5, 64, device="cuda").bfloat16()
    y = ln(x)
    with torch.no_grad():
        ln.bias.add_(1)
    y.backward(torch.ones_like(y))
    assert torch.equal(ln.bias.grad, torch.full_like(ln.bias, 5.0))


@pytest.mark.parametrize("what", ["no bias", "hook", "adapter"])
def test_projections_that_are_not_the_plain_layer(what):
    """The packed-gradient form of the attention needs the package's own projection with a bias; any other one trains as in the
    form without fused blocks.  Two bf16 forms of one network, each within 2 % of the largest value of the true gradient."""
    import copy
    from pccl_b200.models import GPT, GPTConfig
    from pccl_b200.ops import check_status
    torch.manual_seed(10)
    cfg = GPTConfig.tiny()
    model = GPT(cfg, device="cuda")

    class Adapter(torch.nn.Module):
        def __init__(self, inner):
            super().__init__()
            self.inner = inner

        def forward(self, x):
            return self.inner(x) * 1.5

    for blk in model.blocks:
        if what == "no bias":
            blk.qkv.bias = None
        elif what == "hook":
            blk.qkv.register_forward_hook(lambda m, args, out: out * 1.5)
        else:
            blk.qkv = Adapter(blk.qkv)
    plain = copy.deepcopy(model)
    for blk in plain.blocks:
        blk.fuse = False
    ids = torch.randint(0, cfg.vocab_size, (2, cfg.seq_len), device="cuda")
    tgt = ids.roll(-1, 1)
    for m in (model, plain):
        m(ids, tgt).backward()
    check_status("projections")
    for (name, p), q in zip(model.named_parameters(), plain.parameters()):
        if "qkv" in name:
            assert (p.grad.float() - q.grad.float()).abs().max().item() <= 0.04 * q.grad.float().abs().max().item(), name


def test_layer_norm_of_rows_off_the_16_byte_boundaries():
    """Contiguous views that start anywhere are read like aligned ones (same values, same kernel)."""
    from pccl_b200.nn import LayerNorm
    torch.manual_seed(11)
    ln = LayerNorm(64, device="cuda")
    data = torch.randn(3, 20 * 64 + 8, device="cuda").bfloat16()

    def run(shift):
        x, d, g = (data[i, 1:1 + 20 * 64].view(20, 64) if shift else data[i, 1:1 + 20 * 64].clone().view(20, 64) for i in range(3))
        assert (x.data_ptr() % 16 != 0) == shift
        x.requires_grad_(True)
        d.requires_grad_(True)
        s, y = ln.add_norm(x, d, None)
        out = [s, y, ln(x)] + list(torch.autograd.grad([s, y], [x, d, ln.weight, ln.bias], [g, g]))
        return [t.detach() for t in out]

    assert all(torch.equal(a, b) for a, b in zip(run(True), run(False)))


def test_profiler_target_of_the_training_kernels_runs():
    """The documented command, on a small case."""
    import os
    import subprocess
    import sys
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    r = subprocess.run([sys.executable, "-m", "pccl_b200.profile_targets", "train_kernels", "--tokens", "256", "--iters", "1"],
                       cwd=root, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and "ln_bwd_add_colsum" in r.stdout, r.stdout + r.stderr


@pytest.mark.parametrize("batch,seq", [(2, 64), (3, 77), (2, 256)])
@pytest.mark.parametrize("what", ["autograd", "bucket", "frozen", "saved on cpu", "no grad", "grad"])
def test_block_halves_are_their_layers(batch, seq, what, monkeypatch):
    """A block's halves issue the launches of its layers, so loss, logits and every gradient are the same bits as with the layers called
    one by one: up to and above 128 rows, with gradients returned by autograd, written to the bucket, for some parameters or inputs only,
    and with saved tensors that leave the GPU in between."""
    import torch
    from pccl_b200.models import gpt
    cfg = gpt.GPTConfig(n_layer=3, n_head=4, d_model=128, seq_len=seq, vocab_size=264)
    ids = torch.randint(0, 264, (batch, seq), device="cuda")
    got, calls = [], []
    for name in ("attn_in", "mlp_out"):
        half = getattr(gpt, name)
        monkeypatch.setattr(gpt, name, lambda *a, half=half, name=name: (calls.append(name), half(*a))[1])
    for halves in (True, False):
        if not halves:
            assert calls == ["attn_in", "mlp_out"] * 3             # every block of the first run took its halves
            calls.clear()
            monkeypatch.setattr(gpt, "halves_apply", lambda block, x: False)
        torch.manual_seed(3)
        model = gpt.GPT(cfg, device="cuda")
        for p in model.parameters():
            if p.dim() == 1:
                p.data.copy_((torch.randn(p.shape, device="cuda") * 0.3 + (1.0 if p.data.mean() > 0.5 else 0.0)).bfloat16())
        if what == "frozen":
            for m in (model.blocks[0].ln1, model.blocks[1].ln2, model.blocks[1].proj):
                m.requires_grad_(False)
            model.blocks[2].fc2.bias.requires_grad_(False)
        if what == "no grad":
            with torch.no_grad():
                got.append([model.logits(ids)])
            continue
        if what == "grad":
            blk = model.blocks[1]
            wanted = [blk.ln1.weight, blk.qkv.bias, blk.proj.bias, blk.fc1.weight, model.blocks[0].fc2.bias, model.wpe.weight]
            got.append(list(torch.autograd.grad(model(ids, ids.roll(-1, 1)), wanted)))
            continue
        if what == "bucket":
            from pccl_b200.parallel.dp import ShardedDataParallel
            dp = ShardedDataParallel(model, lr=1e-3, heap_bytes=256 << 20)
            loss = dp.train_step(ids, ids.roll(-1, 1)).clone()
            got.append([loss] + [p.main_grad.clone() for p in model.parameters()])
            continue
        hooks = torch.autograd.graph.save_on_cpu() if what == "saved on cpu" else torch.autograd.graph.saved_tensors_hooks(lambda t: t, lambda t: t)
        with hooks:
            loss = model(ids, ids.roll(-1, 1))
        loss.backward()
        got.append([loss.detach()] + [p.grad for p in model.parameters() if p.requires_grad])
    assert not calls
    # the token table's gradient is a sum in no fixed order, and everything else does not depend on it
    for a, b in zip(*got):
        if what != "no grad" and a.shape == (264, 128):
            assert torch.allclose(a.float(), b.float(), rtol=2e-2, atol=1e-4)
        else:
            assert torch.equal(a, b)


@pytest.mark.gpu
@pytest.mark.parametrize("B,T,D,V,extra,bucket", [(1, 1, 8, 3, 0, "none"), (3, 7, 40, 5, 4, "none"), (5, 33, 264, 1001, 1, "new"), (32, 3, 768, 50, 0, "added to"),
                                                  (4, 129, 2048, 517, 2, "new"), (33, 5, 64, 9, 0, "none"), (2, 9, 64, 9, 3, "tok frozen"),
                                                  (2, 9, 64, 9, 3, "pos frozen")])
def test_token_and_position_embedding(B, T, D, V, extra, bucket):
    """One kernel per direction against the layers' own calls: the values are the same, the positions' gradient is a sum in fp32 rounded
    once, the tokens' a sum of bf16 values in no fixed order."""
    from pccl_b200.nn.embedding import _fused, token_position
    from pccl_b200.nn.linear import Embedding
    torch.manual_seed(B + T)
    wte, wpe = Embedding(V, D, device="cuda"), Embedding(T + extra, D, device="cuda")
    ids = torch.randint(-V, V, (B, T + 1), device="cuda")[:, :-1]   # negative ones count from the end
    assert _fused(ids, wte, wpe) == (B <= 32)
    with torch.no_grad():
        want = wte.weight[ids] + wpe.weight[:T][None]
        assert torch.equal(token_position(ids, wte, wpe), want)
    before = [torch.zeros_like(m.weight) for m in (wte, wpe)]
    if bucket in ("new", "added to"):
        for m, b in zip((wte, wpe), before):
            m.weight.main_grad = torch.randn_like(m.weight)
            m.weight._pccl_written = bucket == "added to"
            if bucket == "added to":
                b.copy_(m.weight.main_grad)
    wte.weight.requires_grad_(bucket != "tok frozen")
    wpe.weight.requires_grad_(bucket != "pos frozen")
    y = token_position(ids, wte, wpe)
    assert torch.equal(y, wte.weight[ids] + wpe.weight[:T][None])
    dy = torch.randn(T, B, D, device="cuda").bfloat16().transpose(0, 1)      # not as the kernel reads it
    y.backward(dy)
    pos = dy.float().sum(0).bfloat16()
    want_pos = before[1].clone()
    want_pos[:T] = want_pos[:T] + pos if bucket == "added to" else pos
    tok, mag = before[0].double(), before[0].double().abs()
    tok.index_add_(0, ids.flatten() % V, dy.reshape(-1, D).double())
    mag.index_add_(0, ids.flatten() % V, dy.reshape(-1, D).double().abs())
    n = torch.bincount(ids.flatten() % V, minlength=V)[:, None]
    for m, frozen in ((wte, "tok frozen"), (wpe, "pos frozen")):
        g = getattr(m.weight, "main_grad", None) if bucket in ("new", "added to") else m.weight.grad
        if bucket == frozen:
            assert g is None
        elif m is wte:          # n additions, each off by 2^-8 (half a unit in the last place of 8 bits) of a partial sum, which earlier ones moved
            assert ((g.double() - tok).abs() <= n * 2.0 ** -8 * (1 + 2.0 ** -8) ** n * mag).all()
        else:                   # B fp32 additions in another order may round to the other neighbour: one unit (2^-7) of the sum, one of the total
            assert ((g.float() - want_pos.float()).abs() <= 2.0 ** -7 * ((g - before[1]).float().abs() + g.float().abs()) + B * 2.0 ** -22).all()


@pytest.mark.parametrize("bucket", [False, True])
def test_embedding_gradient_repeats_itself_in_deterministic_mode(bucket):
    """Some 1500 bf16 additions to each of three rows: any other order gives other sums.  The mode counts when the backward pass runs."""
    from pccl_b200.nn.embedding import _fused, token_position
    from pccl_b200.nn.linear import Embedding
    torch.manual_seed(3)
    wte, wpe = Embedding(3, 64, device="cuda"), Embedding(600, 64, device="cuda")
    ids = torch.randint(-3, 3, (8, 577), device="cuda")
    assert _fused(ids, wte, wpe)
    dy = torch.randn(8, 577, 64, device="cuda").bfloat16()
    got, pos = [], []
    for step in range(6):
        if bucket:
            for m in (wte, wpe):
                m.weight.main_grad, m.weight._pccl_written = torch.randn_like(m.weight), False
        wte.weight.grad = wpe.weight.grad = None
        y = token_position(ids, wte, wpe)
        torch.use_deterministic_algorithms(step < 5)
        try:
            y.backward(dy)
        finally:
            torch.use_deterministic_algorithms(False)
        got.append(wte.weight.main_grad if bucket else wte.weight.grad)
        pos.append(wpe.weight.main_grad if bucket else wpe.weight.grad)
    assert all(torch.equal(g, got[0]) for g in got[:5]) and all(torch.equal(p, pos[0]) for p in pos)
    torch.use_deterministic_algorithms(True)
    try:
        want = torch.zeros_like(wte.weight).index_add_(0, ids.flatten() % 3, dy.view(-1, 64))
    finally:
        torch.use_deterministic_algorithms(False)
    assert torch.equal(got[0], want)
