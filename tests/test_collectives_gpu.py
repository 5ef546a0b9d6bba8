"""Hand-written collectives and the interpreter kernel, all ranks emulated on one GPU (one
cooperative launch plays every rank; 'heaps' are buffers of that GPU)."""
import json

import pytest
import torch

pytestmark = pytest.mark.gpu

SIGNAL_OFF = 0            # layout of each emulated heap: [signals 64 KiB | flags 256 KiB | data]
FLAG_OFF = 64 * 1024
DATA_OFF = 512 * 1024
NAMES = {torch.float32: "f32", torch.bfloat16: "bf16", torch.float16: "f16"}


def _heaps(world, data_bytes):
    hs = [torch.zeros(DATA_OFF + data_bytes, dtype=torch.uint8, device="cuda") for _ in range(world)]
    st = [torch.zeros(4, dtype=torch.int32, device="cuda") for _ in range(world)]
    return hs, st


def _view(h, off, n, dtype):
    es = torch.empty((), dtype=dtype).element_size()
    return h[DATA_OFF + off: DATA_OFF + off + n * es].view(dtype)


@pytest.mark.parametrize("world", [2, 4, 8])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("count", [1, 7, 1024, 256 * 1024 + 17])
def test_allreduce_emulated(native, world, dtype, count):
    es = torch.empty((), dtype=dtype).element_size()
    size = (count * es + 255) // 256 * 256
    hs, st = _heaps(world, 2 * size)
    g = torch.Generator(device="cuda").manual_seed(0)
    xs = [torch.randn(count, generator=g, device="cuda").to(dtype) for _ in range(world)]
    for epoch in (1, 2):
        for r in range(world):
            _view(hs[r], 0, count, dtype).copy_(xs[r] * epoch)
        native.emu_collective("allreduce", [h.data_ptr() for h in hs], SIGNAL_OFF, FLAG_OFF, NAMES[dtype], "sum",
                              DATA_OFF, DATA_OFF + size, count, epoch, 0, 1.0, "", 4, 256,
                              torch.cuda.current_stream().cuda_stream, [s.data_ptr() for s in st], [], [], 0)
        torch.cuda.synchronize()
        assert all(s[0].item() == 0 for s in st)
        ref = torch.stack([x.float() * epoch for x in xs]).sum(0)
        tol = 1e-5 * world if dtype == torch.float32 else 0.04 * world
        for r in range(world):
            got = _view(hs[r], size, count, dtype).float()
            assert (got - ref).abs().max().item() <= tol * max(1.0, ref.abs().max().item())


@pytest.mark.parametrize("world", [2, 4, 8])
@pytest.mark.parametrize("dtype,redop", [(torch.float32, "sum"), (torch.bfloat16, "sum"), (torch.bfloat16, "max")])
@pytest.mark.parametrize("count", [2, 1024, 16 * 1024])
def test_allreduce_low_latency_path_emulated(native, world, dtype, redop, count):
    """All-reduce of up to 64 KiB with the flag travelling in the data (8-byte packets {word, launch number}): no barrier,
    out of place and in place, several launches on alternating receive areas."""
    es = torch.empty((), dtype=dtype).element_size()
    size = (count * es + 255) // 256 * 256
    ll_off = DATA_OFF + 2 * size
    hs = [torch.zeros(ll_off + native.LL_LANE_BYTES, dtype=torch.uint8, device="cuda") for _ in range(world)]
    st = [torch.zeros(4, dtype=torch.int32, device="cuda") for _ in range(world)]
    g = torch.Generator(device="cuda").manual_seed(1)
    xs = [torch.randn(count, generator=g, device="cuda").to(dtype) for _ in range(world)]
    for epoch in (1, 2, 3, 4):
        in_place = epoch == 4
        for r in range(world):
            _view(hs[r], 0, count, dtype).copy_(xs[r] * epoch)
        native.emu_collective("allreduce", [h.data_ptr() for h in hs], SIGNAL_OFF, FLAG_OFF, NAMES[dtype], redop,
                              DATA_OFF, DATA_OFF if in_place else DATA_OFF + size, count, epoch, 0, 1.0, "", 4, 256,
                              torch.cuda.current_stream().cuda_stream, [s.data_ptr() for s in st], [], [], 0, 0, 0, ll_off)
        torch.cuda.synchronize()
        assert all(s[0].item() == 0 for s in st), [s.tolist() for s in st]
        stack = torch.stack([(x * epoch).float() for x in xs])
        ref = stack.sum(0) if redop == "sum" else stack.max(0).values
        tol = 1e-5 * world if dtype == torch.float32 else 0.04 * world
        for r in range(world):
            got = _view(hs[r], 0 if in_place else size, count, dtype).float()
            assert (got - ref).abs().max().item() <= tol * max(1.0, ref.abs().max().item()), (epoch, r)
        # the packets of this launch are in the receive area of its parity: the path was taken
        slot = native.LL_LANE_BYTES // 2 // native.MAX_RANKS                      # rank 1's packets in rank 0's area
        first = hs[0][ll_off + (epoch & 1) * (native.LL_LANE_BYTES // 2) + slot:][:8].view(torch.int64)[0].item()
        assert first >> 32 == epoch, "the low-latency path was not taken"


@pytest.mark.parametrize("world", [2, 8])
@pytest.mark.parametrize("redop", ["max", "min"])
def test_allreduce_minmax_in_place(native, world, redop):
    count, dtype = 5000, torch.bfloat16
    hs, st = _heaps(world, 1 << 16)
    g = torch.Generator(device="cuda").manual_seed(1)
    xs = [torch.randn(count, generator=g, device="cuda").to(dtype) for _ in range(world)]
    for r in range(world):
        _view(hs[r], 0, count, dtype).copy_(xs[r])
    native.emu_collective("allreduce", [h.data_ptr() for h in hs], SIGNAL_OFF, FLAG_OFF, "bf16", redop, DATA_OFF, DATA_OFF,
                          count, 1, 1, 1.0, "", 3, 128, torch.cuda.current_stream().cuda_stream,
                          [s.data_ptr() for s in st], [], [], 0)
    torch.cuda.synchronize()
    ref = torch.stack(xs).float().max(0).values if redop == "max" else torch.stack(xs).float().min(0).values
    for r in range(world):
        assert torch.equal(_view(hs[r], 0, count, dtype).float(), ref)


@pytest.mark.parametrize("world", [2, 8])
@pytest.mark.parametrize("count", [16, 4096 + 8, 100003])
def test_reduce_scatter_scale_cast_emulated(native, world, count):
    """Gradient-bucket form: bf16 in, sum over ranks, x 1/world, fp32 out into a plain tensor."""
    dtype = torch.bfloat16
    size = (world * count * 2 + 255) // 256 * 256
    hs, st = _heaps(world, size)
    g = torch.Generator(device="cuda").manual_seed(2)
    xs = [torch.randn(world * count, generator=g, device="cuda").to(dtype) for _ in range(world)]
    outs = [torch.zeros(count, dtype=torch.float32, device="cuda") for _ in range(world)]
    for r in range(world):
        _view(hs[r], 0, world * count, dtype).copy_(xs[r])
    native.emu_collective("reduce_scatter", [h.data_ptr() for h in hs], SIGNAL_OFF, FLAG_OFF, "bf16", "sum", DATA_OFF, 0,
                          count, 1, 2, 1.0 / world, "f32", 4, 256, torch.cuda.current_stream().cuda_stream,
                          [s.data_ptr() for s in st], [], [o.data_ptr() for o in outs], 0)
    torch.cuda.synchronize()
    assert all(s[0].item() == 0 for s in st)
    full = torch.stack([x.float() for x in xs]).sum(0) / world
    for r in range(world):
        assert (outs[r] - full[r * count:(r + 1) * count]).abs().max().item() < 1e-5


@pytest.mark.parametrize("world", [2, 8])
@pytest.mark.parametrize("kind", ["allgather", "alltoall"])
@pytest.mark.parametrize("nbytes", [16, 1000, 64 * 1024 + 48])
def test_allgather_alltoall_emulated(native, world, kind, nbytes):
    size = (world * nbytes + 255) // 256 * 256
    hs, st = _heaps(world, size)
    g = torch.Generator(device="cuda").manual_seed(3)
    n_in = nbytes if kind == "allgather" else world * nbytes
    xs = [torch.randint(0, 255, (n_in,), generator=g, device="cuda", dtype=torch.uint8) for _ in range(world)]
    native.emu_collective(kind, [h.data_ptr() for h in hs], SIGNAL_OFF, FLAG_OFF, "f32", "sum", 0, DATA_OFF, nbytes, 1, 3,
                          1.0, "", 2, 256, torch.cuda.current_stream().cuda_stream, [s.data_ptr() for s in st],
                          [x.data_ptr() for x in xs], [], 0)
    torch.cuda.synchronize()
    assert all(s[0].item() == 0 for s in st)
    for r in range(world):
        got = hs[r][DATA_OFF:DATA_OFF + world * nbytes]
        if kind == "allgather":
            ref = torch.cat(xs)
        else:
            ref = torch.cat([x[r * nbytes:(r + 1) * nbytes] for x in xs])
        assert torch.equal(got, ref)


@pytest.mark.parametrize("algo", ["ring_allreduce", "direct_allreduce", "oneshot_allreduce", "tree_allreduce",
                                  "direct_reduce_scatter", "direct_allgather", "ring_kv_rotation", "alltoall"])
@pytest.mark.parametrize("world,width", [(2, 1), (4, 2)])
def test_interpreter_runs_lowered_programs(native, algo, world, width):
    from pccl_b200.lang import build, to_schedule
    ir = build(algo, world, channels=2)
    doc = json.dumps(to_schedule(ir))
    dtype, n = torch.float32, 3000 + 5
    coll = ir.collective
    n_in = {"allreduce": n, "reduce_scatter": n * world, "allgather": n, "alltoall": n * world}[coll]
    n_out = {"allreduce": n, "reduce_scatter": n, "allgather": n * world, "alltoall": n * world}[coll]
    hs, st = _heaps(world, 16 << 20)
    g = torch.Generator(device="cuda").manual_seed(4)
    xs = [torch.randn(n_in, generator=g, device="cuda") for _ in range(world)]
    ys = [torch.full((n_out,), -5.0, device="cuda") for _ in range(world)]
    for epoch in (0, 1):
        native.emu_program(doc, [h.data_ptr() for h in hs], SIGNAL_OFF, [x.data_ptr() for x in xs],
                           [y.data_ptr() for y in ys], n_in * 4, "f32", width, DATA_OFF + epoch * (8 << 20), 0, epoch,
                           0, [s.data_ptr() for s in st], [], torch.cuda.current_stream().cuda_stream)
        assert all(s[0].item() == 0 for s in st), [s.tolist() for s in st]
        full = torch.stack(xs)
        for r in range(world):
            if coll == "allreduce":
                ref = full.sum(0)
            elif coll == "reduce_scatter":
                ref = full.sum(0)[r * n:(r + 1) * n]
            elif coll == "allgather":
                ref = torch.cat(xs)
            else:
                ref = torch.cat([x[r * n:(r + 1) * n] for x in xs])
            assert (ys[r] - ref).abs().max().item() < 1e-4, (algo, r)


@pytest.mark.parametrize("algo", ["direct_allreduce", "direct_reduce_scatter", "direct_allgather"])
@pytest.mark.parametrize("world,width", [(2, 1), (4, 2), (8, 2)])
def test_interpreter_runs_pull_forms_on_symmetric_buffers(native, algo, world, width):
    """``direct=True``: peers' inputs are read and peers' outputs written in place (same heap offset on every rank), no
    scratch; three launches in a row with changing inputs, so a rank that ran ahead of the barriers would be seen."""
    from pccl_b200.lang import build, to_schedule
    ir = build(algo, world, channels=2, direct=True)
    assert ir.buffers["scratch"] == 0
    doc = json.dumps(to_schedule(ir))
    n = 2048 + 8
    coll = ir.collective
    n_in = {"allreduce": n, "reduce_scatter": n * world, "allgather": n}[coll]
    n_out = {"allreduce": n, "reduce_scatter": n, "allgather": n * world}[coll]
    hs, st = _heaps(world, 4 << 20)
    in_off, out_off = DATA_OFF + (1 << 20), DATA_OFF + (2 << 20)
    g = torch.Generator(device="cuda").manual_seed(14)
    for epoch in range(3):
        xs = [torch.randn(n_in, generator=g, device="cuda") for _ in range(world)]
        for r in range(world):
            _view(hs[r], in_off - DATA_OFF, n_in, torch.float32).copy_(xs[r])
            _view(hs[r], out_off - DATA_OFF, n_out, torch.float32).fill_(-5.0)
        native.emu_program(doc, [h.data_ptr() for h in hs], SIGNAL_OFF, [h.data_ptr() + in_off for h in hs],
                           [h.data_ptr() + out_off for h in hs], n_in * 4, "f32", width, DATA_OFF, 0, epoch,
                           0, [s.data_ptr() for s in st], [], torch.cuda.current_stream().cuda_stream)
        assert all(s[0].item() == 0 for s in st), [s.tolist() for s in st]
        full = torch.stack(xs)
        for r in range(world):
            got = _view(hs[r], out_off - DATA_OFF, n_out, torch.float32)
            ref = full.sum(0) if coll == "allreduce" else (full.sum(0)[r * n:(r + 1) * n] if coll == "reduce_scatter" else torch.cat(xs))
            assert (got - ref).abs().max().item() < 1e-4, (algo, r, epoch)


def test_bounded_wait_returns_timeout_status(native):
    """A wait on a flag nobody sets comes back with ST_TIMEOUT; the context stays usable."""
    flag = torch.zeros(1, dtype=torch.int64, device="cuda")
    st = torch.zeros(4, dtype=torch.int32, device="cuda")
    native.wait_timeout_probe(flag.data_ptr(), 200_000, st.data_ptr(), torch.cuda.current_stream().cuda_stream)
    torch.cuda.synchronize()
    assert st[0].item() == 1
    assert torch.ones(4, device="cuda").sum().item() == 4.0


def test_interpreter_peer_never_arrives(native):
    """Rank 1's streams are left out: rank 0 gives up after its time limit and reports where."""
    from pccl_b200.lang import build, to_schedule
    doc = json.dumps(to_schedule(build("ring_allreduce", 2)))
    hs, st = _heaps(2, 1 << 20)
    xs = [torch.ones(1024, device="cuda") for _ in range(2)]
    ys = [torch.zeros(1024, device="cuda") for _ in range(2)]
    native.emu_program(doc, [h.data_ptr() for h in hs], SIGNAL_OFF, [x.data_ptr() for x in xs], [y.data_ptr() for y in ys],
                       4096, "f32", 1, DATA_OFF, 0, 0, 100_000, [s.data_ptr() for s in st], [1],
                       torch.cuda.current_stream().cuda_stream)
    assert st[0][0].item() == 1 and st[1][0].item() == 0
    assert torch.ones(4, device="cuda").sum().item() == 4.0


@pytest.mark.parametrize("world", [2, 4, 8])
@pytest.mark.parametrize("kind,redop", [("allreduce_fp8", "sum"), ("allreduce_fp8", "max"), ("reduce_scatter_fp8", "sum")])
def test_fp8_block_scaled_reduce_emulated(native, world, kind, redop):
    """Block-scaled fp8 all-reduce / reduce-scatter: dequantise, accumulate in fp32, requantise with a fresh scale."""
    from pccl_b200.ops.gemm import dequant_rows, quant_rows
    shard_blocks = 24
    n = 128 * shard_blocks * world            # elements of the whole vector
    g = torch.Generator(device="cuda").manual_seed(33)
    xs = [(torch.randn(n // 128, 128, generator=g, device="cuda") * (1 + r)).bfloat16() for r in range(world)]
    qs = [quant_rows(x) for x in xs]
    q_in, s_in = DATA_OFF, DATA_OFF + n
    q_out, s_out = s_in + (n // 128) * 4, s_in + (n // 128) * 4 + n
    hs = [torch.zeros(s_out + (n // 128) * 4 + 256, dtype=torch.uint8, device="cuda") for _ in range(world)]
    st = [torch.zeros(4, dtype=torch.int32, device="cuda") for _ in range(world)]
    for r in range(world):
        hs[r][q_in:q_in + n] = qs[r][0].view(-1)
        hs[r][s_in:s_in + (n // 128) * 4].view(torch.float32)[:] = qs[r][1].view(-1)
    count = n if kind == "allreduce_fp8" else n // world
    native.emu_collective(kind, [h.data_ptr() for h in hs], SIGNAL_OFF, FLAG_OFF, "e4m3", redop, q_in, q_out, count, 1, 2, 1.0, "",
                          4, 256, torch.cuda.current_stream().cuda_stream, [s.data_ptr() for s in st], [], [], 0, s_in, s_out)
    torch.cuda.synchronize()
    assert all(s[0].item() == 0 for s in st), [s.tolist() for s in st]
    vals = torch.stack([dequant_rows(q, s) for q, s in qs])       # [world, n/128, 128] exact inputs
    ref = vals.sum(0) if redop == "sum" else vals.amax(0)
    for r in range(world):
        if kind == "allreduce_fp8":
            oq = hs[r][q_out:q_out + n].view(n // 128, 128)
            os_ = hs[r][s_out:s_out + (n // 128) * 4].view(torch.float32).view(n // 128, 1)
            want = ref
        else:
            m = n // world
            oq = hs[r][q_out:q_out + m].view(m // 128, 128)
            os_ = hs[r][s_out:s_out + (m // 128) * 4].view(torch.float32).view(m // 128, 1)
            want = ref[r * shard_blocks:(r + 1) * shard_blocks]
        # the fresh scale is the block maximum over 448, and the payload is the e4m3 rounding of value / scale
        assert torch.allclose(os_.view(-1), want.abs().amax(-1) / 448.0, rtol=1e-5, atol=0)
        got = dequant_rows(oq, os_)
        assert (got - want).abs().max().item() <= 0.0625 * want.abs().max().item() + 1e-6
        want_q = (want / os_).to(torch.float8_e4m3fn).float()
        assert (oq.view(torch.float8_e4m3fn).float() - want_q).abs().max().item() <= 32.0     # at most one e4m3 step at the top of the range


# ---------------------------------------------------------------------------------------------
# fused collective + GEMM kernels, ranks emulated on one GPU
# ---------------------------------------------------------------------------------------------
@pytest.mark.parametrize("world,tail", [(2, -1), (4, -1), (2, 0), (2, 2), (2, 100), (4, 5)])
def test_ag_gemm_emulated(native, world, tail):
    """`tail`: tiles at the end of the tile order that the copy CTAs compute after sending their rows (-1: cost model,
    0: none, a number beyond the tile count: all of them)."""
    M_local, K, N = 256, 512, 520
    M = M_local * world
    g = torch.Generator(device="cuda").manual_seed(9)
    xs = [(torch.randn(M_local, K, generator=g, device="cuda") * 0.5).bfloat16() for _ in range(world)]
    ws = [(torch.randn(N, K, generator=g, device="cuda") * 0.1).bfloat16() for _ in range(world)]
    x_off = DATA_OFF
    ready_off = DATA_OFF + M * K * 2
    heaps = [torch.zeros(ready_off + 4096, dtype=torch.uint8, device="cuda") for _ in range(world)]
    st = [torch.zeros(4, dtype=torch.int32, device="cuda") for _ in range(world)]
    outs = [torch.zeros(M, N, dtype=torch.bfloat16, device="cuda") for _ in range(world)]
    ctas = 148 // world
    for epoch in (1, 2):
        for r in range(world):
            full = heaps[r][x_off:x_off + M * K * 2].view(torch.bfloat16).view(M, K)
            full.zero_()
            full[r * M_local:(r + 1) * M_local] = xs[r] * epoch
        native.emu_ag_gemm([h.data_ptr() for h in heaps], FLAG_OFF, x_off, M, N, K, [w.data_ptr() for w in ws], K,
                           [o.data_ptr() for o in outs], N, ready_off, epoch, 4, ctas,
                           [s.data_ptr() for s in st], 0, torch.cuda.current_stream().cuda_stream, tail)
        torch.cuda.synchronize()
        assert all(s[0].item() == 0 for s in st), [s.tolist() for s in st]
        X = torch.cat(xs).float() * epoch
        for r in range(world):
            ref = X @ ws[r].float().t()
            assert (outs[r].float() - ref).abs().max().item() < 0.03 * max(1.0, ref.abs().max().item())
            gathered = heaps[r][x_off:x_off + M * K * 2].view(torch.bfloat16).view(M, K)
            assert torch.equal(gathered.float(), X)


@pytest.mark.parametrize("world,M_local", [(2, 128), (2, 256), (4, 128), (2, 512)])
def test_gemm_rs_emulated(native, world, M_local):
    K, N = 448, 512     # 256 rows per rank and an even CTA count take the CTA-pair pipeline (whole rows staged per tile)
    M = M_local * world
    g = torch.Generator(device="cuda").manual_seed(10)
    ys = [(torch.randn(M, K, generator=g, device="cuda") * 0.5).bfloat16() for _ in range(world)]
    ws = [(torch.randn(N, K, generator=g, device="cuda") * 0.1).bfloat16() for _ in range(world)]
    stage_bytes = world * M_local * N * 2
    n_flags = world * (M_local // 128) * (N // 256)
    heaps = [torch.zeros(DATA_OFF + stage_bytes + n_flags * 8, dtype=torch.uint8, device="cuda") for _ in range(world)]
    st = [torch.zeros(4, dtype=torch.int32, device="cuda") for _ in range(world)]
    outs = [torch.zeros(M_local, N, dtype=torch.bfloat16, device="cuda") for _ in range(world)]
    for epoch in (1, 2):
        native.emu_gemm_rs([h.data_ptr() for h in heaps], [y.data_ptr() for y in ys], K, [w.data_ptr() for w in ws], K,
                           [o.data_ptr() for o in outs], N, M, N, K, DATA_OFF, DATA_OFF + stage_bytes, epoch, 148 // world,
                           [s.data_ptr() for s in st], 0, torch.cuda.current_stream().cuda_stream)
        torch.cuda.synchronize()
        assert all(s[0].item() == 0 for s in st), [s.tolist() for s in st]
        total = sum(ys[r].float() @ ws[r].float().t() for r in range(world))
        for r in range(world):
            ref = total[r * M_local:(r + 1) * M_local]
            assert (outs[r].float() - ref).abs().max().item() < 0.03 * max(1.0, ref.abs().max().item())
        for y in ys:
            y.mul_(0.5)


@pytest.mark.parametrize("world,quant_out", [(2, False), (4, False), (2, True)])
def test_ag_gemm_fp8_emulated(native, world, quant_out):
    from pccl_b200.ops.gemm import dequant_blocks, dequant_rows, quant_blocks, quant_rows
    M_local, K, N = 256, 1024, 512
    M = M_local * world
    g = torch.Generator(device="cuda").manual_seed(19)
    xs = [(torch.randn(M_local, K, generator=g, device="cuda") * 0.5).bfloat16() for _ in range(world)]
    ws = [quant_blocks((torch.randn(N, K, generator=g, device="cuda") * 0.1).bfloat16()) for _ in range(world)]
    x_off = DATA_OFF
    xs_off = x_off + M * K
    ready_off = xs_off + M * (K // 128) * 4
    heaps = [torch.zeros(ready_off + 4096, dtype=torch.uint8, device="cuda") for _ in range(world)]
    st = [torch.zeros(4, dtype=torch.int32, device="cuda") for _ in range(world)]
    outs = [torch.zeros(M, N, dtype=torch.bfloat16, device="cuda") for _ in range(world)]
    oq = [torch.zeros(M, N, dtype=torch.uint8, device="cuda") for _ in range(world)]
    os_ = [torch.zeros(M, N // 128, dtype=torch.float32, device="cuda") for _ in range(world)]
    ctas = 148 // world
    for epoch in (1, 2):
        X = []
        for r in range(world):
            q, s = quant_rows((xs[r].float() * epoch).bfloat16())
            X.append(dequant_rows(q, s))
            fq = heaps[r][x_off:x_off + M * K].view(M, K)
            fs = heaps[r][xs_off:xs_off + M * (K // 128) * 4].view(torch.float32).view(M, K // 128)
            fq.zero_()
            fs.zero_()
            fq[r * M_local:(r + 1) * M_local] = q
            fs[r * M_local:(r + 1) * M_local] = s
        native.ag_gemm_fp8(None, [h.data_ptr() for h in heaps], FLAG_OFF, x_off, xs_off, M, N, K, [w[0].data_ptr() for w in ws], K,
                           [w[1].data_ptr() for w in ws], K // 128, [] if quant_out else [o.data_ptr() for o in outs], N,
                           [o.data_ptr() for o in oq] if quant_out else [], [o.data_ptr() for o in os_] if quant_out else [], N,
                           0, native.GEMM_GELU_INPLACE if quant_out else 0, ready_off, epoch, 4, ctas, 0,
                           [s.data_ptr() for s in st], 0, torch.cuda.current_stream().cuda_stream)
        torch.cuda.synchronize()
        assert all(s[0].item() == 0 for s in st), [s.tolist() for s in st]
        X = torch.cat(X)
        for r in range(world):
            ref = X @ dequant_blocks(*ws[r]).t()
            if quant_out:
                ref = torch.nn.functional.gelu(ref, approximate="tanh")
                got = dequant_rows(oq[r], os_[r])
                # e4m3 keeps 3 mantissa bits: half a unit in the last place of the block maximum
                assert (got - ref).abs().max().item() <= 0.07 * max(1.0, ref.abs().max().item())
                assert torch.allclose(os_[r], ref.view(M, N // 128, 128).abs().amax(-1) / 448.0, rtol=2e-2, atol=1e-6)
            else:
                assert (outs[r].float() - ref).abs().max().item() < 0.02 * max(1.0, ref.abs().max().item())
            gq = heaps[r][x_off:x_off + M * K].view(M, K)
            gs = heaps[r][xs_off:xs_off + M * (K // 128) * 4].view(torch.float32).view(M, K // 128)
            assert torch.equal(dequant_rows(gq, gs), X)


@pytest.mark.parametrize("world", [2, 4])
def test_ag_gemm_mx8_emulated(native, world):
    """All-gather -> GEMM on the hardware block-scaled pipeline: e4m3 rows and UE8M0 scale bytes are gathered."""
    from pccl_b200.ops.gemm import dequant_blocks, dequant_rows, quant_blocks_mx, quant_rows_mx, ue8m0_to_float
    M_local, K, N = 256, 1024, 640
    M = M_local * world
    g = torch.Generator(device="cuda").manual_seed(29)
    xs = [(torch.randn(M_local, K, generator=g, device="cuda") * (0.5 + r)).bfloat16() for r in range(world)]
    ws = [quant_blocks_mx((torch.randn(N, K, generator=g, device="cuda") * 0.1).bfloat16()) for _ in range(world)]
    x_off = DATA_OFF
    xs_off = x_off + M * K
    ready_off = xs_off + M * (K // 128)
    heaps = [torch.zeros(ready_off + 4096, dtype=torch.uint8, device="cuda") for _ in range(world)]
    st = [torch.zeros(4, dtype=torch.int32, device="cuda") for _ in range(world)]
    outs = [torch.zeros(M, N, dtype=torch.bfloat16, device="cuda") for _ in range(world)]
    ctas = 148 // world
    for epoch in (1, 2):
        X = []
        for r in range(world):
            q, s = quant_rows_mx((xs[r].float() * epoch).bfloat16())
            X.append(dequant_rows(q, ue8m0_to_float(s)))
            fq = heaps[r][x_off:x_off + M * K].view(M, K)
            fs = heaps[r][xs_off:xs_off + M * (K // 128)].view(M, K // 128)
            fq.zero_()
            fs.zero_()
            fq[r * M_local:(r + 1) * M_local] = q
            fs[r * M_local:(r + 1) * M_local] = s
        native.ag_gemm_fp8(None, [h.data_ptr() for h in heaps], FLAG_OFF, x_off, xs_off, M, N, K, [w[0].data_ptr() for w in ws], K,
                           [w[1].data_ptr() for w in ws], K // 128, [o.data_ptr() for o in outs], N, [], [], 0, 0, 0, ready_off, epoch,
                           4, ctas, 0, [s.data_ptr() for s in st], 0, torch.cuda.current_stream().cuda_stream, True)
        torch.cuda.synchronize()
        assert all(s[0].item() == 0 for s in st), [s.tolist() for s in st]
        X = torch.cat(X)
        for r in range(world):
            ref = X @ dequant_blocks(ws[r][0], ue8m0_to_float(ws[r][1])).t()
            assert (outs[r].float() - ref).abs().max().item() < 0.02 * max(1.0, ref.abs().max().item())
            gs = heaps[r][xs_off:xs_off + M * (K // 128)].view(M, K // 128)
            assert torch.equal(dequant_rows(heaps[r][x_off:x_off + M * K].view(M, K), ue8m0_to_float(gs)), X)


@pytest.mark.parametrize("world,M_local", [(2, 128), (2, 256), (4, 128)])
def test_gemm_rs_fp8_emulated(native, world, M_local):
    from pccl_b200.ops.gemm import dequant_blocks, dequant_rows, quant_blocks, quant_rows
    K, N = 512, 512
    M = M_local * world
    g = torch.Generator(device="cuda").manual_seed(20)
    ys = [quant_rows((torch.randn(M, K, generator=g, device="cuda") * 0.5).bfloat16()) for _ in range(world)]
    ws = [quant_blocks((torch.randn(N, K, generator=g, device="cuda") * 0.1).bfloat16()) for _ in range(world)]
    stage_bytes = world * M_local * N * 2
    n_flags = world * (M_local // 128) * (N // 256)
    heaps = [torch.zeros(DATA_OFF + stage_bytes + n_flags * 8, dtype=torch.uint8, device="cuda") for _ in range(world)]
    st = [torch.zeros(4, dtype=torch.int32, device="cuda") for _ in range(world)]
    outs = [torch.zeros(M_local, N, dtype=torch.bfloat16, device="cuda") for _ in range(world)]
    total = sum(dequant_rows(*ys[r]) @ dequant_blocks(*ws[r]).t() for r in range(world))
    for epoch in (1, 2):
        native.gemm_rs_fp8(None, [h.data_ptr() for h in heaps], [y[0].data_ptr() for y in ys], K, [y[1].data_ptr() for y in ys], K // 128,
                           [w[0].data_ptr() for w in ws], K, [w[1].data_ptr() for w in ws], K // 128, [o.data_ptr() for o in outs], N,
                           M, N, K, DATA_OFF, DATA_OFF + stage_bytes, epoch, 148 // world, [s.data_ptr() for s in st], 0,
                           torch.cuda.current_stream().cuda_stream)
        torch.cuda.synchronize()
        assert all(s[0].item() == 0 for s in st), [s.tolist() for s in st]
        for r in range(world):
            ref = total[r * M_local:(r + 1) * M_local]
            assert (outs[r].float() - ref).abs().max().item() < 0.03 * max(1.0, ref.abs().max().item())
        for o in outs:
            o.zero_()


# ---------------------------------------------------------------------------------------------
# MoE kernels
# ---------------------------------------------------------------------------------------------
def test_fp8_quantisers_match_reference(native):
    from pccl_b200.ops.moe import quant_fp8_blocks, quant_fp8_rows
    torch.manual_seed(3)
    x = (torch.randn(300, 1024, device="cuda") * 3).bfloat16()
    q, s = quant_fp8_rows(x)
    xf = x.float().view(300, 8, 128)
    ref_s = xf.abs().amax(-1) / 448.0
    assert torch.allclose(s, ref_s, rtol=1e-6, atol=0)
    ref_q = (xf / ref_s[..., None]).to(torch.float8_e4m3fn).view(300, 1024).float()
    got_q = q.view(torch.float8_e4m3fn).float()
    # the kernel multiplies by a reciprocal: a value that sits on a rounding boundary may land one
    # fp8 step away from the divide-then-round reference, never further
    assert (got_q == ref_q).float().mean().item() > 0.999
    assert ((got_q - ref_q).abs() <= 0.0625 * ref_q.abs() + 2 ** -9).all()
    w = (torch.randn(256, 384, device="cuda")).bfloat16()
    qw, sw = quant_fp8_blocks(w)
    wf = w.float().view(2, 128, 3, 128).permute(0, 2, 1, 3)
    ref_sw = wf.abs().amax((-1, -2)) / 448.0
    assert torch.allclose(sw, ref_sw, rtol=1e-6, atol=0)
    deq = qw.view(torch.float8_e4m3fn).float().view(2, 128, 3, 128) * sw[:, None, :, None]
    assert (deq.view(256, 384) - w.float()).abs().max().item() <= 0.07 * w.float().abs().max().item()


@pytest.mark.parametrize("N,gelu", [(384, False), (512, False), (768, True)])
def test_grouped_gemm_matches_per_group_reference(native, N, gelu):
    """The CTA-pair kernel with the operands exchanged (N = 384: the last weight tile reaches past the group's features), whose tiles end where a group's rows end (group sizes around and off the multiples of 16 and 256)."""
    from pccl_b200.ops import check_status
    from pccl_b200.ops.moe import grouped_gemm
    torch.manual_seed(4)
    K = 512
    sizes = [130, 0, 257, 5, 128, 64, 513, 16, 300, 1]
    off = torch.tensor([0] + list(torch.tensor(sizes).cumsum(0)), dtype=torch.int32, device="cuda")
    total = int(off[-1])
    a = (torch.randn(total + 200, K, device="cuda") * 0.5).bfloat16()
    b = (torch.randn(len(sizes) * N, K, device="cuda") * 0.1).bfloat16()
    out = torch.full((total + 200, N), 7.0, device="cuda", dtype=torch.bfloat16)
    grouped_gemm(a, b, off, N, out=out, gelu=gelu)
    check_status("grouped gemm")
    for g, n in enumerate(sizes):
        lo = int(off[g])
        ref = a[lo:lo + n].float() @ b[g * N:(g + 1) * N].float().t()
        if gelu:
            ref = torch.nn.functional.gelu(ref, approximate="tanh")
        assert (out[lo:lo + n].float() - ref).abs().max().item() < 0.05 if n else True
    assert torch.all(out[total:] == 7.0)        # rows past the last group are untouched


@pytest.mark.parametrize("N,K,b_t", [(384, 512, False), (392, 192, False), (256, 512, True), (136, 192, True), (648, 200, True)])
def test_grouped_gemm_gelu_forms(native, N, K, b_t):
    """GELU side output and GELU-backward epilogue of the grouped kernel, weights as [n, K] and [K, n]: feature counts off the
    256-row tiles (136, 392, 648), a K that ends inside a k-block (200: laid out anew for the [K, n] form), groups around the
    multiples of 16 and 256.  fp32 sums of <= 512 terms and one bf16 rounding: 2^-8 of the value and of the largest."""
    from pccl_b200.ops import check_status
    from pccl_b200.ops.moe import grouped_gemm
    torch.manual_seed(5)
    sizes = [17, 0, 257, 1, 256, 15]
    off = torch.tensor([0] + list(torch.tensor(sizes).cumsum(0)), dtype=torch.int32, device="cuda")
    total, G = int(off[-1]), len(sizes)
    a = (torch.randn(total + 40, K, device="cuda") * 0.5).bfloat16()
    b = (torch.randn((G * K, N) if b_t else (G * N, K), device="cuda") * 0.1).bfloat16()
    pre_in = torch.randn(total + 40, N, device="cuda").bfloat16()
    act = torch.full((total + 40, N), 7.0, device="cuda", dtype=torch.bfloat16)
    pre, d = act.clone(), act.clone()
    grouped_gemm(a, b, off, N, out=pre, gelu_out=act, b_t=b_t)
    grouped_gemm(a, b, off, N, out=d, dgelu=pre_in, b_t=b_t)
    check_status("grouped gemm")
    for g, n in enumerate(sizes):
        s = slice(int(off[g]), int(off[g]) + n)
        w = b[g * K:(g + 1) * K].double() if b_t else b[g * N:(g + 1) * N].double().t()
        ref = (a[s].double() @ w).requires_grad_(True)
        x = pre_in[s].double().requires_grad_(True)
        gx, = torch.autograd.grad(torch.nn.functional.gelu(x, approximate="tanh").sum(), x)
        for got, want in ((pre[s], ref), (act[s], torch.nn.functional.gelu(ref, approximate="tanh")), (d[s], ref * gx)):
            assert (got.double() - want).abs().le(2 ** -8 * want.abs() + 1e-5).all()
    assert all((t[total:] == 7.0).all() for t in (pre, act, d))                     # rows past the last group are untouched


@pytest.mark.parametrize("sizes", [[130, 0, 257, 1, 64, 63, 65, 0], [0, 0, 5], [512]])
@pytest.mark.parametrize("M,N", [(256, 512), (136, 328)])
def test_grouped_weight_gradients(native, M, N, sizes):
    """Group ends inside and at the edges of a k-block, empty groups, feature counts off the tiles; the rows past the last group
    hold NaN (they are uninitialised memory in use) and must not be read into any sum."""
    from pccl_b200.ops import check_status
    from pccl_b200.ops.moe import grouped_wgrad
    torch.manual_seed(6)
    off = torch.tensor([0] + list(torch.tensor(sizes).cumsum(0)), dtype=torch.int32, device="cuda")
    total = int(off[-1])
    ops = [torch.randn(total + 70, f, device="cuda").bfloat16() for f in (M, N, N, M)]
    for t in ops:
        t[total:] = float("nan")
    d0, d1 = grouped_wgrad(*ops, off)
    check_status("grouped weight gradients")
    for d, a, b in ((d0, ops[0], ops[1]), (d1, ops[2], ops[3])):
        d = d.view(len(sizes), a.shape[1], b.shape[1])
        for g, n in enumerate(sizes):
            s = slice(int(off[g]), int(off[g]) + n)
            ref = a[s].double().t() @ b[s].double()
            assert (d[g].double() - ref).abs().le(2 ** -8 * ref.abs() + 1e-4).all()


@pytest.mark.parametrize("T,blocks", [(64, 8), (20, 8), (300, 2)])      # one token per group of threads, groups without a token, many trips
def test_moe_dispatch_combine_emulated(native, T, blocks):
    """Two emulated ranks: fp8 dispatch lands in the right rows with the right scales; combine pulls
    rows back from both ranks and weights them."""
    world, H, Kt, epr = 2, 256, 2, 2
    cap = max(512, world * T * Kt)
    q_off, s_off, y_off = DATA_OFF, DATA_OFF + cap * H, DATA_OFF + cap * H + cap * (H // 128) * 4
    heaps = [torch.zeros(y_off + cap * H * 2, dtype=torch.uint8, device="cuda") for _ in range(world)]
    st = [torch.zeros(4, dtype=torch.int32, device="cuda") for _ in range(world)]
    g = torch.Generator(device="cuda").manual_seed(5)
    xs = [(torch.randn(T, H, generator=g, device="cuda") * 2).bfloat16() for _ in range(world)]
    ids = [torch.randint(0, world * epr, (T, Kt), generator=g, device="cuda", dtype=torch.int32) for _ in range(world)]
    # every (rank, token, k) gets a unique row on its destination: rank r uses rows r*T*Kt + t*Kt + k
    rows = [(torch.arange(T * Kt, device="cuda", dtype=torch.int32) + r * T * Kt).view(T, Kt).contiguous() for r in range(world)]
    probs = [torch.rand(T, Kt, generator=g, device="cuda") for _ in range(world)]
    outs = [torch.zeros(T, H, dtype=torch.bfloat16, device="cuda") for _ in range(world)]
    stream = torch.cuda.current_stream().cuda_stream
    native.moe_exchange("dispatch", None, [h.data_ptr() for h in heaps], FLAG_OFF, T, H, Kt, epr, q_off, s_off, y_off, 1, 0,
                        [x.data_ptr() for x in xs], [i.data_ptr() for i in ids], [r.data_ptr() for r in rows], [], [],
                        [s.data_ptr() for s in st], blocks, 0, stream)
    torch.cuda.synchronize()
    assert all(s[0].item() == 0 for s in st)
    from pccl_b200.ops.moe import quant_fp8_rows
    for r in range(world):
        q_ref, s_ref = quant_fp8_rows(xs[r])
        for t in range(0, T, 7):
            for k in range(Kt):
                d, row = int(ids[r][t, k]) // epr, int(rows[r][t, k])
                got_q = heaps[d][q_off + row * H: q_off + (row + 1) * H]
                got_s = heaps[d][s_off + row * (H // 128) * 4: s_off + (row + 1) * (H // 128) * 4].view(torch.float32)
                assert torch.equal(got_q, q_ref[t]) and torch.equal(got_s, s_ref[t])
    # expert outputs: fill y on both ranks with a known function of (rank, row)
    ys = []
    for d in range(world):
        y = heaps[d][y_off:y_off + cap * H * 2].view(torch.bfloat16).view(cap, H)
        y.copy_((torch.randn(cap, H, generator=g, device="cuda")).bfloat16())
        ys.append(y)
    native.moe_exchange("combine", None, [h.data_ptr() for h in heaps], FLAG_OFF, T, H, Kt, epr, q_off, s_off, y_off, 2, 0,
                        [], [i.data_ptr() for i in ids], [r.data_ptr() for r in rows], [p.data_ptr() for p in probs],
                        [o.data_ptr() for o in outs], [s.data_ptr() for s in st], blocks, 0, stream)
    torch.cuda.synchronize()
    assert all(s[0].item() == 0 for s in st)
    for r in range(world):
        ref = torch.zeros(T, H, device="cuda")
        for k in range(Kt):
            d = (ids[r][:, k] // epr).long()
            picked = torch.stack([ys[int(d[t])][int(rows[r][t, k])] for t in range(T)]).float()
            ref += probs[r][:, k, None] * picked
        assert (outs[r].float() - ref).abs().max().item() < 0.05


@pytest.mark.parametrize("T,blocks", [(64, 8), (20, 8), (300, 2)])
def test_moe_deduplicated_exchange_emulated(native, T, blocks):
    """Two emulated ranks, four assignments per token over four experts: most tokens have several assignments on one
    rank.  The dispatch sends the row once per rank and tells the others where it is; the conversion to bf16 fills every
    row; the ranks add up each token's weighted expert outputs locally and the combine pulls one row per rank."""
    world, H, Kt, epr = 2, 256, 4, 2
    cap = max(1024, world * T * Kt)
    G = H // 128
    q_off = DATA_OFF
    s_off = q_off + cap * H
    y_off = s_off + cap * G * 4
    alias_off = y_off + cap * H * 2
    group_off = alias_off + cap * 4
    z_off = group_off + cap * 64
    heaps = [torch.zeros(z_off + cap * H * 2, dtype=torch.uint8, device="cuda") for _ in range(world)]
    st = [torch.zeros(4, dtype=torch.int32, device="cuda") for _ in range(world)]
    g = torch.Generator(device="cuda").manual_seed(15)
    xs = [(torch.randn(T, H, generator=g, device="cuda") * 2).bfloat16() for _ in range(world)]
    ids = [torch.randint(0, world * epr, (T, Kt), generator=g, device="cuda", dtype=torch.int32) for _ in range(world)]
    ids[0][3, 1] = -1                                   # a dropped assignment takes no part in any group
    rows = [(torch.arange(T * Kt, device="cuda", dtype=torch.int32) + r * T * Kt).view(T, Kt).contiguous() for r in range(world)]
    probs = [torch.rand(T, Kt, generator=g, device="cuda") for _ in range(world)]
    outs = [torch.zeros(T, H, dtype=torch.bfloat16, device="cuda") for _ in range(world)]
    stream = torch.cuda.current_stream().cuda_stream
    hp = [h.data_ptr() for h in heaps]
    native.moe_exchange("dispatch", None, hp, FLAG_OFF, T, H, Kt, epr, q_off, s_off, y_off, 1, 0,
                        [x.data_ptr() for x in xs], [i.data_ptr() for i in ids], [r.data_ptr() for r in rows], [], [],
                        [s.data_ptr() for s in st], blocks, 0, stream, alias_off=alias_off, group_off=group_off, z_off=z_off,
                        gate=[p.data_ptr() for p in probs], dedupe=True)
    torch.cuda.synchronize()
    assert all(s[0].item() == 0 for s in st)
    from pccl_b200.ops.moe import quant_fp8_rows
    n_rows = torch.tensor([world * T * Kt], dtype=torch.int32, device="cuda")
    sent = skipped = 0
    xb = []
    for d in range(world):
        out = torch.zeros(cap, H, dtype=torch.bfloat16, device="cuda")
        native.moe_dequant(heaps[d].data_ptr() + q_off, heaps[d].data_ptr() + s_off, out.data_ptr(), n_rows.data_ptr(), cap, H, stream,
                           alias=heaps[d].data_ptr() + alias_off)
        xb.append(out)
    torch.cuda.synchronize()
    for r in range(world):
        q_ref, s_ref = quant_fp8_rows(xs[r])
        deq = (q_ref.view(torch.float8_e4m3fn).float().view(T, G, 128) * s_ref.view(T, G, 1)).view(T, H).bfloat16()
        for t in range(T):
            seen = set()
            for k in range(Kt):
                e = int(ids[r][t, k])
                if e < 0:
                    continue
                d, row = e // epr, int(rows[r][t, k])
                payload = heaps[d][q_off + row * H: q_off + (row + 1) * H]
                if d in seen:
                    skipped += 1
                    assert not payload.any()                      # never sent
                else:
                    sent += 1
                    assert torch.equal(payload, q_ref[t])
                seen.add(d)
                assert torch.equal(xb[d][row], deq[t]), (r, t, k)   # every row is there after the conversion
    assert skipped > T and sent > T
    ys = []
    for d in range(world):
        y = heaps[d][y_off:y_off + cap * H * 2].view(torch.bfloat16).view(cap, H)
        y.copy_((torch.randn(cap, H, generator=g, device="cuda")).bfloat16())
        ys.append(y)
        native.moe_reduce_groups(heaps[d].data_ptr() + y_off, heaps[d].data_ptr() + z_off, heaps[d].data_ptr() + alias_off,
                                 heaps[d].data_ptr() + group_off, n_rows.data_ptr(), cap, H, stream)
    native.moe_exchange("combine", None, hp, FLAG_OFF, T, H, Kt, epr, q_off, s_off, y_off, 2, 0,
                        [], [i.data_ptr() for i in ids], [r.data_ptr() for r in rows], [p.data_ptr() for p in probs],
                        [o.data_ptr() for o in outs], [s.data_ptr() for s in st], blocks, 0, stream, alias_off=alias_off,
                        group_off=group_off, z_off=z_off, dedupe=True)
    torch.cuda.synchronize()
    assert all(s[0].item() == 0 for s in st)
    for r in range(world):
        ref = torch.zeros(T, H, device="cuda")
        for t in range(T):
            for k in range(Kt):
                e = int(ids[r][t, k])
                if e >= 0:
                    ref[t] += probs[r][t, k] * ys[e // epr][int(rows[r][t, k])].float()
        assert (outs[r].float() - ref).abs().max().item() < 0.06, r


def test_moe_layer_world_of_one_matches_dense_reference(native):
    from pccl_b200.engine import Engine
    from pccl_b200.ops import check_status
    from pccl_b200.ops.moe import MoEExchange
    torch.manual_seed(6)
    T, H, F, E, Kt = 256, 512, 256, 8, 2
    eng = Engine(0, 1)
    eng.initEngine("cuda", heap_bytes=512 << 20)
    moe = MoEExchange(eng, T, H, E, Kt)
    x = torch.randn(T, H, device="cuda").bfloat16()
    logits = torch.randn(T, E, device="cuda")
    w1 = (torch.randn(E * F, H, device="cuda") * 0.05).bfloat16()
    w2 = (torch.randn(E * H, F, device="cuda") * 0.05).bfloat16()
    out = moe.forward(x, logits, w1, w2)
    check_status("moe")
    ids, probs = MoEExchange.route(logits, Kt)
    ref = torch.zeros(T, H, device="cuda")
    xq = x.float().view(T, H // 128, 128)
    sc = xq.abs().amax(-1, keepdim=True) / 448.0
    xd = ((xq / sc).to(torch.float8_e4m3fn).float() * sc).view(T, H).bfloat16().float()   # what the experts see
    for e in range(E):
        h = torch.nn.functional.gelu(xd @ w1[e * F:(e + 1) * F].float().t(), approximate="tanh").bfloat16().float()
        y = (h @ w2[e * H:(e + 1) * H].float().t()).bfloat16().float()
        for k in range(Kt):
            m = (ids[:, k] == e)
            ref[m] += probs[m, k, None] * y[m]
    assert (out.float() - ref).abs().max().item() < 0.03 * max(1.0, ref.abs().max().item())
    del moe, eng


def test_moe_route_and_plan_kernels_match_tensor_ops(native):
    from pccl_b200.engine import Engine
    from pccl_b200.ops.moe import MoEExchange
    torch.manual_seed(8)
    T, H, E, Kt = 1000, 256, 64, 6
    eng = Engine(0, 1); eng.initEngine("cuda", heap_bytes=256 << 20)
    moe = MoEExchange(eng, T, H, E, Kt)
    logits = torch.randn(T, E, device="cuda")
    ids, probs, plan = moe.route_and_plan(logits)
    ref_ids, ref_probs = MoEExchange.route(logits, Kt)
    ref_plan = moe.plan(ref_ids)
    assert torch.equal(ids, ref_ids)
    assert torch.allclose(probs, ref_probs, rtol=1e-4, atol=1e-7)
    assert torch.equal(plan["row_off"], ref_plan["row_off"])
    # rows are a permutation within each expert's segment: same multiset per expert, all distinct
    rows, ref_rows = plan["rows"].view(-1).long(), ref_plan["rows"].view(-1).long()
    assert rows.unique().numel() == rows.numel()
    off = plan["row_off"].long()
    flat = ids.view(-1).long()
    assert ((rows >= off[flat]) & (rows < off[flat + 1])).all()
    assert torch.equal(rows.sort().values, ref_rows.sort().values)
    del moe, eng


@pytest.mark.parametrize("algo", ["ring_allreduce", "direct_allreduce", "direct_reduce_scatter", "direct_allgather", "alltoall"])
def test_engine_regop_exeop_on_a_cuda_engine_with_alternating_widths(native, algo):
    """The public path initEngine("cuda") -> regOp -> exeOp on a world of one: the program is materialised per width,
    every (program, width) pair gets its own signal words and launch count, the scratch half alternates per launch, and
    the interpreter kernel runs it on the GPU.  A world of one keeps every wait inside one launch."""
    from pccl_b200.engine import Engine
    from pccl_b200.lang import build
    eng = Engine(0, 1)
    eng.initEngine("cuda", heap_bytes=512 << 20)       # the default 256 MiB workspace and some room for tensors
    eng.regOp("op", build(algo, 1, channels=2))
    n = 3 * 8192 + 16
    for it, width in enumerate([1, 4, 1, 4, 2, 4]):
        x = torch.arange(n, device="cuda", dtype=torch.float32) + it
        y = torch.full((n,), -1.0, device="cuda")
        eng.exeOp("op", x, y, width=width, check=True)
        assert torch.equal(y, x), (algo, it, width)
    st = eng.stats()
    assert st["ops"]["op"]["launches"] == 6 and st["device"] == "cuda" and st["signals_used"] > 0
    # a symmetric (heap) tensor works as well, and in place
    z = eng.symmetric_tensor((n,), torch.float32)
    z.copy_(torch.arange(n, device="cuda", dtype=torch.float32))
    if algo.endswith("allreduce"):
        eng.exeOp("op", z, width=2, check=True)
        assert torch.equal(z, torch.arange(n, device="cuda", dtype=torch.float32))
    del eng


def test_resident_executor_takes_queued_launches_without_a_kernel_launch_each(native):
    """startResident -> enqueue x N -> wait: the interpreter kernel stays on the GPU and takes its work from a queue in
    pinned host memory (a world of one keeps every wait inside the one kernel).  It leaves by itself when idle and is
    started again by the next submission."""
    import time
    from pccl_b200.engine import Engine
    from pccl_b200.lang import build
    eng = Engine(0, 1)
    eng.initEngine("cuda", heap_bytes=512 << 20)
    eng.regOp("ar", build("ring_allreduce", 1, channels=2))
    eng.regOp("ag", build("direct_allgather", 1, channels=1))
    eng.start_resident(width=2)
    n = 64 * 1024
    xs = [torch.arange(n, device="cuda", dtype=torch.float32) + i for i in range(24)]
    ys = [torch.full((n,), -1.0, device="cuda") for _ in range(24)]
    torch.cuda.current_stream().synchronize()
    t0 = time.perf_counter()
    tickets = [eng.enqueue("ar" if i % 3 else "ag", xs[i], ys[i], sync_inputs=False) for i in range(24)]
    eng.wait(tickets[-1], timeout_ms=20000)
    per_op_us = (time.perf_counter() - t0) / 24 * 1e6
    for i in range(24):
        assert torch.equal(ys[i], xs[i]), i
    st = eng.stats()
    assert st["resident_ops"] == 24 and st["resident_kernel_launches"] >= 1
    first_launches = st["resident_kernel_launches"]
    assert first_launches <= 3, st            # not one launch per operation
    assert eng.check_status(0)[0] == 0
    # idle: the kernel leaves (a device-wide synchronize returns), the next submission brings it back
    time.sleep(0.1)
    torch.cuda.synchronize()
    y = torch.zeros(n, device="cuda")
    eng.wait(eng.enqueue("ar", xs[3], y), timeout_ms=20000)
    assert torch.equal(y, xs[3])
    assert eng.stats()["resident_kernel_launches"] > first_launches
    eng.stop_resident()
    eng.exeOp("ar", xs[5], y, check=True)          # the launch-per-call path still works afterwards
    assert torch.equal(y, xs[5])
    print(f"resident executor: {per_op_us:.1f} us per queued operation (host clock, 24 operations)")
    del eng


def test_moe_layer_backward_matches_dense_reference(native):
    """The expert-parallel layer as an autograd node (world of one): gradients of the input, the gate logits and both
    expert weights against a dense fp32 reference that sees the same e4m3 round trips as the kernels."""
    from pccl_b200.engine import Engine
    from pccl_b200.ops import check_status
    from pccl_b200.ops.moe import MoEExchange
    from pccl_b200.parallel.ep import _MoEFn
    torch.manual_seed(16)
    T, H, Fd, E, Kt = 256, 512, 256, 8, 2
    eng = Engine(0, 1)
    eng.initEngine("cuda", heap_bytes=512 << 20)
    moe = MoEExchange(eng, T, H, E, Kt)
    x = torch.randn(T, H, device="cuda").bfloat16().requires_grad_(True)
    logits = torch.randn(T, E, device="cuda").requires_grad_(True)
    w1 = (torch.randn(E * Fd, H, device="cuda") * 0.05).bfloat16().requires_grad_(True)
    w2 = (torch.randn(E * H, Fd, device="cuda") * 0.05).bfloat16().requires_grad_(True)
    g = (torch.randn(T, H, device="cuda") * 0.1).bfloat16()
    out = _MoEFn.apply(x, logits, w1, w2, moe)
    out.backward(g)
    check_status("moe backward")

    def e4m3_round_trip(t):      # what a row looks like after the dispatch (1 x 128 blocks)
        q = t.view(t.shape[0], -1, 128)
        sc = (q.abs().amax(-1, keepdim=True) / 448.0).clamp_min(1e-30)
        return ((q / sc).to(torch.float8_e4m3fn).float() * sc).view_as(t)

    xr = x.detach().float().requires_grad_(True)
    lr = logits.detach().float().requires_grad_(True)
    w1r, w2r = w1.detach().float().requires_grad_(True), w2.detach().float().requires_grad_(True)
    pf = torch.softmax(lr, -1)
    p, ids = pf.topk(Kt, -1)
    xs = xr + (e4m3_round_trip(xr.detach()) - xr.detach())            # straight-through: forward sees the quantised rows
    ref = torch.zeros(T, H, device="cuda")
    for e in range(E):
        y = torch.nn.functional.gelu(xs @ w1r[e * Fd:(e + 1) * Fd].t(), approximate="tanh") @ w2r[e * H:(e + 1) * H].t()
        for k in range(Kt):
            m = (ids[:, k] == e).float()[:, None]
            ref = ref + m * p[:, k, None] * y
    ref.backward(g.float())
    assert (out.float() - ref.detach()).abs().max().item() < 0.03 * max(1.0, ref.abs().max().item())
    for got, want, name, tol in ((x.grad, xr.grad, "dx", 0.08), (logits.grad, lr.grad, "dlogits", 0.08), (w1.grad, w1r.grad, "dw1", 0.08),
                                 (w2.grad, w2r.grad, "dw2", 0.08)):
        err = (got.float() - want).abs().max().item()
        assert err <= tol * max(1e-6, want.abs().max().item()), (name, err, want.abs().max().item())
    del moe, eng


def test_run_time_compiled_program_launches_and_mixes_with_the_interpreter(native):
    """JitOp on a world of one: the generated kernel (NVRTC -> cubin -> driver launch) gives the program's result, at two
    widths and two sizes, interleaved with interpreter launches of the same program on the same lane."""
    from pccl_b200.engine import Engine
    from pccl_b200.jit import JitOp
    from pccl_b200.lang import build
    eng = Engine(0, 1)
    eng.initEngine("cuda", heap_bytes=512 << 20)
    eng.regOp("ar", build("ring_allreduce", 1, channels=2))
    eng.regOp("ag", build("direct_allgather", 1, channels=1))
    ar, ag = JitOp(eng, "ar"), JitOp(eng, "ag")
    for it, (n, width) in enumerate([(4096, 1), (4096, 2), (3 * 8192 + 16, 2), (4096, 1)]):
        x = torch.arange(n, device="cuda", dtype=torch.float32) + it
        y = torch.full((n,), -1.0, device="cuda")
        ar(x, y, width=width)
        torch.cuda.synchronize()
        assert torch.equal(y, x), (it, n, width)
        y.fill_(-1)
        eng.exeOp("ar", x, y, width=width, check=True)          # the interpreter on the same signal range and lane
        assert torch.equal(y, x)
        g = torch.zeros(n, device="cuda")
        ag(x, g)
        torch.cuda.synchronize()
        assert torch.equal(g, x)
    assert ar.compiled == 3 and eng.check_status(0)[0] == 0      # (4096, 1) was compiled once
    xb = torch.randn(8192, device="cuda").bfloat16()
    yb = torch.zeros_like(xb)
    ar(xb, yb, width=2)
    torch.cuda.synchronize()
    assert torch.equal(xb, yb)
    del ar, ag, eng


@pytest.mark.parametrize("tokens,ff", [(256, 320), (768, 64), (256, 328), (384, 320), (768, 4672)])       # the last one: tiles of 224 columns
def test_tp_mlp_world_of_one_matches_fp64(native, tokens, ff):
    """The MLP as one node (GELU, its derivative and the biases in the fused kernels' epilogues), and the layer-by-layer form that
    a d_ff off the multiples of 32 (328) or rows off the multiples of 256 (384) take.  Against fp64; up to four bf16 roundings
    in a row (2^-9 at most, 0.17 % rms each) give 0.4 % in norm."""
    from pccl_b200.engine import Engine
    from pccl_b200.ops import check_status
    from pccl_b200.parallel.tp import TensorParallelMLP
    torch.manual_seed(8)
    d = 512
    eng = Engine(0, 1)
    eng.initEngine("cuda", 512 << 20)
    mlp = TensorParallelMLP(eng, tokens, d, ff)
    mlp.fc1.bias.data.normal_(0, 0.5)
    mlp.fc2.bias.data.normal_(0, 0.5)
    mlp.fc1.weight.data.mul_(3)
    x = torch.randn(tokens, d, device="cuda").bfloat16().requires_grad_(True)
    dz = torch.randn(tokens, d, device="cuda").bfloat16()
    params = [x] + list(mlp.parameters())
    z = mlp(x)
    grads = torch.autograd.grad(z, params, dz)
    again = torch.autograd.grad(mlp(x), params, dz)
    check_status("tp mlp")
    assert all(torch.equal(g, h) for g, h in zip(grads, again))
    p64 = [p.detach().double().requires_grad_(True) for p in params]
    names = ["x"] + [n for n, _ in mlp.named_parameters()]
    q = dict(zip(names, p64))
    h = torch.nn.functional.gelu(q["x"] @ q["fc1.weight"].t() + q["fc1.bias"], approximate="tanh")
    z64 = h @ q["fc2.weight"].t() + q["fc2.bias"]
    g64 = torch.autograd.grad(z64, p64, dz.double())
    for got, want in zip((z,) + tuple(grads), (z64,) + tuple(g64)):
        assert ((got.double() - want).norm() / want.norm()).item() < 8e-3
    del mlp, eng


@pytest.mark.parametrize("what", ["fp32", "unaligned", "scalar"])
def test_row_parallel_bias_that_the_kernel_cannot_add(native, what):
    """A bias of another type, alignment or shape than the epilogue loads is added by torch, as a layer of its own would."""
    from pccl_b200.engine import Engine
    from pccl_b200.ops import check_status
    from pccl_b200.parallel.tp import RowParallelLinear
    torch.manual_seed(12)
    eng = Engine(0, 1)
    eng.initEngine("cuda", 256 << 20)
    layer = RowParallelLinear(eng, 256, 64, 256)
    bias = {"fp32": torch.randn(256, device="cuda"), "unaligned": torch.randn(257, device="cuda").bfloat16()[1:],
            "scalar": torch.randn(1, device="cuda").bfloat16()}[what]
    h = torch.randn(256, 64, device="cuda").bfloat16().requires_grad_(True)
    layer.bias = None
    plain = layer(h).detach()
    layer.bias = torch.nn.Parameter(bias)
    z = layer(h)
    assert torch.equal(z, plain + bias)
    z.sum().backward()
    check_status("row parallel bias")
    assert torch.equal(layer.bias.grad, (torch.full_like(bias, 256.0) if bias.numel() > 1 else torch.full_like(bias, 65536.0)))
    del layer, eng


@pytest.mark.parametrize("what", ["wrapped", "patched", "global hook"])
def test_tp_mlp_with_layers_that_are_not_plain(native, what):
    """A layer that is wrapped, has a forward of its own or is seen by a global hook is called, not passed by."""
    from pccl_b200.engine import Engine
    from pccl_b200.ops import check_status
    from pccl_b200.parallel.tp import TensorParallelMLP
    torch.manual_seed(13)
    eng = Engine(0, 1)
    eng.initEngine("cuda", 256 << 20)
    mlp = TensorParallelMLP(eng, 256, 256, 64)
    x = torch.randn(256, 256, device="cuda").bfloat16()
    plain = torch.nn.functional.gelu(mlp.fc1(x), approximate="tanh")
    calls = []
    handle = None
    if what == "wrapped":
        class Wrapped(torch.nn.Module):
            def __init__(self, inner):
                super().__init__()
                self.inner = inner

            def forward(self, x):
                calls.append(1)
                return self.inner(x)

        mlp.fc1 = Wrapped(mlp.fc1)
    elif what == "patched":
        forward = mlp.fc2.forward
        mlp.fc2.forward = lambda h: (calls.append(1), forward(h))[1]
    else:
        handle = torch.nn.modules.module.register_module_forward_hook(lambda m, args, out: calls.append(type(m).__name__))
    try:
        z = mlp(x)
    finally:
        if handle is not None:
            handle.remove()
    assert calls and (what != "global hook" or set(calls) == {"TensorParallelMLP", "ColumnParallelLinear", "RowParallelLinear"})
    assert torch.equal(z, mlp.fc2(plain))
    check_status("tp mlp")
    del mlp, eng


@pytest.mark.parametrize("N,shift", [(30, 0), (2, 0), (300, 0), (64, 2), (256, 1)])
def test_grouped_gemm_into_unaligned_or_odd_outputs(native, N, shift):
    """Feature counts that are no multiple of four and outputs off the 8-byte boundaries: the row-major form of the grouped kernel.
    fp32 sums of 128 terms and one bf16 rounding."""
    from pccl_b200.ops import check_status
    from pccl_b200.ops.moe import grouped_gemm
    torch.manual_seed(6)
    K, sizes = 128, [130, 0, 5, 257]
    off = torch.tensor([0] + list(torch.tensor(sizes).cumsum(0)), dtype=torch.int32, device="cuda")
    total = int(off[-1])
    a = (torch.randn(total + 3, K, device="cuda") * 0.5).bfloat16()
    b = (torch.randn(len(sizes) * N, K, device="cuda") * 0.1).bfloat16()
    ld = (N + shift + 7) // 8 * 8
    store = torch.full((total + 3, ld), 7.0, device="cuda", dtype=torch.bfloat16)
    out = store[:, shift:shift + N]
    grouped_gemm(a, b, off, N, out=out, gelu=N == 300)
    check_status("grouped gemm")
    for g, n in enumerate(sizes):
        lo = int(off[g])
        ref = a[lo:lo + n].double() @ b[g * N:(g + 1) * N].double().t()
        if N == 300:
            ref = torch.nn.functional.gelu(ref, approximate="tanh")
        assert ((out[lo:lo + n].double() - ref).abs() <= 2 ** -8 * ref.abs() + (2e-3 if N == 300 else 1e-5)).all()      # hardware tanh
    assert (store[:, :shift] == 7.0).all() and (store[:, shift + N:] == 7.0).all() and (store[total:] == 7.0).all()


@pytest.mark.parametrize("E,Kt", [(8, 3), (33, 4), (1024, 8)])
def test_moe_route_with_nan_and_infinite_logits_stays_in_range(native, E, Kt):
    """Logits of a diverged model still give experts that exist; a row of good logits beside them is not disturbed."""
    from pccl_b200._native import C
    from pccl_b200.ops.moe import MoEExchange
    torch.manual_seed(14)
    T = 70
    logits = torch.randn(T, E, device="cuda")
    logits[1:20] = float("nan")
    logits[1:10, 2] = 1.0
    logits[20:30, 1] = float("inf")
    logits[30:40] = -float("inf")
    ids = torch.full((T, Kt), -7, dtype=torch.int32, device="cuda")
    pos, probs = ids.clone(), torch.empty((T, Kt), device="cuda")
    counts = torch.zeros(E, dtype=torch.int32, device="cuda")
    C.moe_route(logits.data_ptr(), ids.data_ptr(), probs.data_ptr(), pos.data_ptr(), counts.data_ptr(), T, E, Kt,
                torch.cuda.current_stream().cuda_stream)
    assert ((ids >= 0) & (ids < E)).all()
    assert torch.equal(counts.long(), torch.bincount(ids.view(-1).long(), minlength=E))
    assert ((pos >= 0) & (pos < counts[ids.long()])).all()
    good = [0] + list(range(40, T))
    ref_ids, ref_probs = MoEExchange.route(logits[good], Kt)
    assert torch.equal(ids[good], ref_ids) and torch.allclose(probs[good], ref_probs, rtol=1e-4, atol=1e-7)


@pytest.mark.parametrize("world,M_local,N,w_t", [(2, 256, 520, False), (4, 256, 96, True), (2, 512, 320, True), (2, 4352, 512, False)])
def test_ag_gemm_gelu_forms_emulated(native, world, M_local, N, w_t):
    """Bias and GELU, and the GELU-backward form with its column sums, over the gathered rows of several ranks; 4352 rows per rank
    are a second block of 16 tile rows.  One bf16 rounding (2^-8), fp32 sums of 64 terms; column sums of unrounded values."""
    K = 64
    M = M_local * world
    g = torch.Generator(device="cuda").manual_seed(15)
    def rand(*shape, scale=1.0):
        return (torch.randn(*shape, generator=g, device="cuda") * scale).bfloat16()
    xs = [rand(M_local, K, scale=0.5) for _ in range(world)]
    ws = [rand(K, N, scale=0.1) if w_t else rand(N, K, scale=0.1) for _ in range(world)]
    bias = [rand(N) for _ in range(world)]
    pre_in = [rand(M, N, scale=1.5) for _ in range(world)]
    ready_off = DATA_OFF + M * K * 2
    heaps = [torch.zeros(ready_off + 4096, dtype=torch.uint8, device="cuda") for _ in range(world)]
    st = [torch.zeros(4, dtype=torch.int32, device="cuda") for _ in range(world)]
    for r in range(world):
        heaps[r][DATA_OFF:ready_off].view(torch.bfloat16).view(M, K)[r * M_local:(r + 1) * M_local] = xs[r]
    pre, act, dpre = ([torch.full((M, N), 7.0, dtype=torch.bfloat16, device="cuda") for _ in range(world)] for _ in range(3))
    parts = [torch.empty((M + 31) // 32 * N, device="cuda") for _ in range(world)]
    sums = [torch.full((N,), 9.0, dtype=torch.bfloat16, device="cuda") for _ in range(world)]
    at = lambda ts: [t.data_ptr() for t in ts]  # noqa: E731
    ctas = (148 // world) & ~1

    def run(out, epoch, **kw):
        native.emu_ag_gemm(at(heaps), FLAG_OFF, DATA_OFF, M, N, K, at(ws), ws[0].stride(0), at(out), N, ready_off, epoch, 4, ctas, at(st), 0,
                           torch.cuda.current_stream().cuda_stream, b_mn=w_t, **kw)

    run(pre, 1, flags=native.GEMM_GELU | native.GEMM_GELU_FULL, bias=at(bias), d2=at(act))
    forms = [(pre, lambda p, r: p + bias[r].double()), (act, lambda p, r: torch.nn.functional.gelu(p + bias[r].double(), approximate="tanh"))]
    if N % 32 == 0:
        def back(p, r):
            x = pre_in[r].double().requires_grad_(True)
            gx, = torch.autograd.grad(torch.nn.functional.gelu(x, approximate="tanh").sum(), x)
            return p * gx
        run(dpre, 2, flags=native.GEMM_DGELU, d2=at(pre_in), parts=at(parts), colsum=at(sums))
        forms.append((dpre, back))
    torch.cuda.synchronize()
    assert all(s[0].item() == 0 for s in st), [s.tolist() for s in st]
    X = torch.cat(xs).double()
    for r in range(world):
        prod = X @ (ws[r].double() if w_t else ws[r].double().t())
        for got, want in forms:
            ref = want(prod, r)
            assert ((got[r].double() - ref).abs() <= 2 ** -8 * ref.abs() + 1e-5).all()
        if N % 32 == 0:
            ref = back(prod, r)
            assert ((sums[r].double() - ref.sum(0)).abs() <= 2 ** -8 * ref.sum(0).abs() + 1e-5 * ref.abs().sum(0)).all()


@pytest.mark.parametrize("world,M_local,w_t", [(2, 128, False), (2, 256, True), (4, 256, False), (2, 4352, False)])
def test_gemm_rs_bias_emulated(native, world, M_local, w_t):
    """Every rank adds its bias to its own rows, once; 4352 rows per rank are a second block of 16 tile rows.  The peers' partial sums
    are rounded to bf16 on the way: 2^-8 of each, and of the result."""
    K, N = 64, 512
    M = M_local * world
    g = torch.Generator(device="cuda").manual_seed(16)
    def rand(*shape, scale=1.0):
        return (torch.randn(*shape, generator=g, device="cuda") * scale).bfloat16()
    ys = [rand(M, K, scale=0.5) for _ in range(world)]
    ws = [rand(K, N, scale=0.1) if w_t else rand(N, K, scale=0.1) for _ in range(world)]
    bias = [rand(N) for _ in range(world)]
    stage_bytes = world * M_local * N * 2
    n_flags = world * (M_local // 128) * (N // 256)
    heaps = [torch.zeros(DATA_OFF + stage_bytes + n_flags * 8, dtype=torch.uint8, device="cuda") for _ in range(world)]
    st = [torch.zeros(4, dtype=torch.int32, device="cuda") for _ in range(world)]
    outs = [torch.zeros(M_local, N, dtype=torch.bfloat16, device="cuda") for _ in range(world)]
    at = lambda ts: [t.data_ptr() for t in ts]  # noqa: E731
    native.emu_gemm_rs(at(heaps), at(ys), K, at(ws), ws[0].stride(0), at(outs), N, M, N, K, DATA_OFF, DATA_OFF + stage_bytes, 1, 148 // world,
                       at(st), 0, torch.cuda.current_stream().cuda_stream, b_mn=w_t, bias=at(bias))
    torch.cuda.synchronize()
    assert all(s[0].item() == 0 for s in st), [s.tolist() for s in st]
    parts = [ys[r].double() @ (ws[r].double() if w_t else ws[r].double().t()) for r in range(world)]
    for r in range(world):
        rows = slice(r * M_local, (r + 1) * M_local)
        ref = sum(p[rows] for p in parts) + bias[r].double()
        spread = sum(p[rows].abs() for p in parts) + ref.abs()
        assert ((outs[r].double() - ref).abs() <= 2 ** -8 * spread + 1e-5).all()


@pytest.mark.parametrize("T,H,E,topk", [(40, 128, 8, 1), (41, 2176, 8, 3), (300, 1024, 16, 8), (97, 7168, 32, 8), (33, 16512, 4, 4)])
def test_moe_exchange_group_sizes(native, T, H, E, topk):
    """Tokens handled by groups of 64 and of 256 threads (the launch picks by tokens per block): the same bytes, scales and combined
    rows; the gate gradients add up in another order (fp32 sums of H products: 1e-5 of the sum of magnitudes)."""
    from pccl_b200.engine import Engine
    from pccl_b200.ops import check_status
    from pccl_b200.ops.moe import MoEExchange
    torch.manual_seed(T)
    eng = Engine(0, 1)
    cap = 2 * T * topk + 256
    eng.initEngine("cuda", 2 * cap * (H * 5 + H // 32 + 256) + (640 << 20))
    x, logits = torch.randn(T, H, device="cuda").bfloat16(), torch.randn(T, E, device="cuda")
    y = torch.randn(cap, H, device="cuda").bfloat16()
    got = []
    for blocks in (1, 148):
        ex = MoEExchange(eng, T, H, E, topk, blocks=blocks)
        if not got:
            ids, probs, plan = ex.route_and_plan(logits)
        n = T * topk
        ex.dispatch(x, ids, plan)
        plain = (ex.recv_q[:n].clone(), ex.recv_s[:n].clone())
        ex.dispatch(x, ids, plan, probs=probs)
        scaled = (ex.recv_q[:n].clone(), ex.recv_s[:n].clone())
        ex.y.copy_(y[:ex.cap])
        got.append(plain + scaled + (ex.combine(ids, probs, plan), ex.combine_dot(x, ids, plan)))
        check_status("moe exchange")
    for a, b in zip(got[0][:5], got[1][:5]):
        assert torch.equal(a, b)
    rows = plan["rows"].long()
    products = x.double()[:, None, :] * y.double()[rows]
    for g in got:
        assert ((g[5].double() - products.sum(-1)).abs() <= 1e-5 * products.abs().sum(-1)).all()
    want = (probs.double()[:, :, None] * y.double()[rows]).sum(1)
    assert ((got[0][4].double() - want).abs() <= 2 ** -8 * want.abs() + 1e-4).all()


@pytest.mark.parametrize("T,E,topk", [(1, 1, 1), (9, 31, 2), (64, 32, 8), (33, 100, 4), (17, 256, 8), (5, 1024, 8)])
def test_moe_route_backward(native, T, E, topk):
    """One to 32 experts per lane, experts that fill no lane count, against autograd in fp64 (fp32 sums of E terms: 1e-5 of the largest
    gradient); logits far apart and a plain combine without weights."""
    from pccl_b200.engine import Engine
    from pccl_b200.ops.moe import MoEExchange
    torch.manual_seed(E)
    eng = Engine(0, 1)
    eng.initEngine("cuda", 640 << 20)
    ex = MoEExchange(eng, T, 128, E, topk)
    logits = torch.randn(T, E, device="cuda") * 6
    ids, probs, plan = ex.route_and_plan(logits)
    dp = torch.randn(T, topk, device="cuda")
    l64 = logits.double().requires_grad_(True)
    (torch.softmax(l64, -1).gather(1, ids.long()) * dp.double()).sum().backward()
    got = ex.route_backward(logits, ids, dp)
    assert (got.double() - l64.grad).abs().max().item() <= 1e-5 * max(1e-3, l64.grad.abs().max().item())
    ex.y.copy_(torch.randn(ex.y.shape, device="cuda"))
    assert torch.equal(ex.combine(ids, None, plan), ex.combine(ids, torch.ones_like(probs), plan))


@pytest.mark.parametrize("T,H,E,topk,drop", [(1, 128, 8, 1, 0), (7, 128, 8, 2, 5), (41, 2176, 8, 3, 0), (130, 1024, 16, 8, 40), (97, 7168, 32, 8, 0), (9, 16512, 4, 4, 3)])
def test_moe_deliver_in_a_world_of_one(native, T, H, E, topk, drop):
    """The rows that one kernel writes are those of dispatch and conversion, bit for bit, plain and scaled, for widths off the 256 values of
    a warp, blocks of zeros and infinities, and with assignments dropped by row and by expert; nothing else is written."""
    from pccl_b200.engine import Engine
    from pccl_b200.ops import check_status
    from pccl_b200.ops.moe import MoEExchange
    torch.manual_seed(T)
    eng = Engine(0, 1)
    cap = 2 * T * topk + 256
    eng.initEngine("cuda", 2 * cap * (H * 5 + H // 32 + 256) + (640 << 20))
    ex = MoEExchange(eng, T, H, E, topk)
    x = torch.randn(T, H, device="cuda").bfloat16() * torch.logspace(-8, 8, T, device="cuda")[:, None].bfloat16()
    x[T // 2, :128] = 0
    if T > 8:
        x[3, 5] = float("inf")
    ids, probs, plan = ex.route_and_plan(torch.randn(T, E, device="cuda"))
    rows = plan["rows"].flatten().long()
    if drop:
        plan["rows"].view(-1)[:drop] = -1
        ids.view(-1)[-1] = -1
    kept = torch.ones(T * topk, dtype=torch.bool, device="cuda")
    if drop:
        kept[:drop] = False
        kept[-1] = False
    for p in (None, probs):
        ex.dispatch(x, ids, plan, probs=p)
        want = ex.received(plan)
        got = ex.deliver(x, ids, plan, probs=p, out=torch.full((ex.cap, H), 3.0, device="cuda").bfloat16())
        assert torch.equal(got[rows[kept]].view(torch.int16), want[rows[kept]].view(torch.int16))
        rest = torch.ones(ex.cap, dtype=torch.bool, device="cuda")
        rest[rows[kept]] = False
        assert (got[rest] == 3.0).all()
    check_status("moe deliver")


def test_moe_received_after_a_pass_in_a_world_of_one(native):
    """``received`` (and ``experts``) behind ``forward`` or a layer's pass give that pass's rows and not those of an earlier dispatch; rows past
    the count are left alone; rows that are gone are refused."""
    from pccl_b200.engine import Engine
    from pccl_b200.ops.moe import MoEExchange
    torch.manual_seed(12)
    T, H, F, E, topk = 33, 256, 128, 8, 2
    eng = Engine(0, 1)
    eng.initEngine("cuda", 640 << 20)
    ex, fresh = MoEExchange(eng, T, H, E, topk), MoEExchange(eng, T, H, E, topk)
    w1, w2 = (torch.randn(E * F, H, device="cuda") * 0.1).bfloat16(), (torch.randn(E * H, F, device="cuda") * 0.1).bfloat16()
    logits, old, x = torch.randn(T, E, device="cuda"), torch.randn(T, H, device="cuda").bfloat16(), torch.randn(T, H, device="cuda").bfloat16()
    ids, probs, plan = ex.route_and_plan(logits)
    n = T * topk

    def want(t):                                       # one row per expert, whatever order the routing gave its tokens
        fresh.dispatch(t, ids, plan)
        return fresh.received(plan)[:n]

    def rows_of(t, p):                                 # the same by token: a pass of its own may place an expert's tokens in another order
        return t[p["rows"].flatten().long()]

    ex.dispatch(old, ids, plan)
    with torch.no_grad():
        ex.forward(x, logits, w1, w2)
    for mode in (torch.no_grad, torch.inference_mode):
        with mode():
            ex.deliver(x, ids, plan, out=ex.x_bf16)
            out = torch.full((ex.cap, H), 3.0, device="cuda").bfloat16()
            assert ex.received(plan, out) is out
            assert torch.equal(out[:n], want(x)) and (out[n:] == 3.0).all()
            assert torch.equal(rows_of(ex.received(plan), plan), rows_of(want(x), plan))
            ex.experts(w1, w2, plan)
            fresh.dispatch(x, ids, plan)
            fresh.experts(w1, w2, plan)
            assert torch.equal(ex.y[:n], fresh.y[:n])
    ex.dispatch(old, ids, plan)
    assert torch.equal(ex.received(plan)[:n], want(old))
    with torch.no_grad():                              # forward's own routing: the multiset of rows is the new tokens'
        ex.forward(x, logits, w1, w2)
    got = ex.received(plan)[:n].float().sum(1).sort().values
    assert torch.equal(got, want(x).float().sum(1).sort().values)
    kept = ex.deliver(old, ids, plan)
    assert torch.equal(ex.received(plan)[:n], want(old))
    kept.add_(1)
    with pytest.raises(RuntimeError, match="gone"):
        ex.received(plan)
    ex.deliver(x, ids, plan)
    with pytest.raises(RuntimeError, match="gone"):
        ex.received(plan)
    ex.dispatch(x, ids, plan)
    assert torch.equal(ex.received(plan)[:n], want(x))
