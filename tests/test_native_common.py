import json
import os

import pytest
import torch


def test_hex_hash_time(native):
    u = native.utils
    blob = bytes(range(256))
    assert u.decode_hex(u.encode_hex(blob)) == blob
    assert u.encode_hex(b"\x00\xff\x10") == "00ff10"
    with pytest.raises(RuntimeError):
        u.decode_hex("abc")
    with pytest.raises(RuntimeError):
        u.decode_hex("zz")
    assert u.fnv1a("") == 14695981039346656037
    assert u.fnv1a("a") == 0xaf63dc4c8601ec8c
    t0 = u.now_nanos(); assert u.now_nanos() >= t0 > 1_600_000_000 * 10**9
    assert len(u.launch_timestamp().split("-")) == 3


def test_env_registry(native):
    L = native.utils.LaunchEnvironments
    opts = L.listOpt()
    for name in ("PCCL_LOG_LEVEL", "PCCL_WORKSPACE_MB", "PCCL_SPIN_LIMIT", "PCCL_TRANSPORT", "PCCL_IB_DEVICE"):
        assert name in opts
    assert L.getEnv("PCCL_SURELY_NOT_SET") == ""
    L.registerOpt("PCCL_TEST_OPTION", "made by a test")
    assert "PCCL_TEST_OPTION" in L.listOpt() and L.helpOf("PCCL_TEST_OPTION") == "made by a test"
    L.setOverride("PCCL_TEST_OPTION", "42")
    assert L.getEnv("PCCL_TEST_OPTION") == "42"
    assert L.getEnv("PATH") == os.environ["PATH"]


def test_json_and_logging(native):
    u = native.utils
    doc = {"a": [1, 2.5, True, None, "x\n\"y\""], "b": {"c": -7, "d": 1e-3}}
    assert json.loads(u.json_roundtrip(json.dumps(doc))) == doc
    with pytest.raises(RuntimeError):
        u.json_roundtrip("{\"a\": [1, 2}")
    before = u.log_count("error")
    u.log("error", "test message 123")
    assert u.log_count("error") == before + 1
    with open(u.log_path()) as f:
        assert "test message 123" in f.read()


def test_type_registry(native):
    u = native.utils
    a = u.register_type(3, "cpu"); b = u.register_type(3, "cuda")
    assert u.register_type(3, "cpu") == a and a != b
    assert "cuda" in u.type_names(3)
    u.set_compatible("cuda_interpreter", 1, "bf16")
    assert u.executors_for(1, "bf16") == ["cuda_interpreter"]


def test_cpu_number_formats(native):
    u = native.utils
    for v in (0.0, 1.0, -2.5, 3.140625, 1e-3, 65504.0, 448.0, -448.0, 0.015625):
        assert u.bf16_roundtrip(v) == torch.tensor(v).bfloat16().float().item()
        assert u.f16_roundtrip(v) == torch.tensor(v).half().float().item()
    if hasattr(torch, "float8_e4m3fn"):
        xs = torch.linspace(-500, 500, 4001).tolist() + [2 ** -9, 2 ** -10 * 1.5, 0.0019]
        for v in xs:
            want = torch.tensor(v).clamp(-448, 448).to(torch.float8_e4m3fn).float().item()
            assert u.e4m3_roundtrip(v) == want, v


@pytest.mark.parametrize("dtype,name", [(torch.float32, "f32"), (torch.bfloat16, "bf16"), (torch.float16, "f16"),
                                        (torch.int32, "i32"), (torch.float64, "f64")])
@pytest.mark.parametrize("op", ["sum", "max", "min"])
def test_cpu_reduce(native, dtype, name, op):
    g = torch.Generator().manual_seed(1)
    a = (torch.randn(1000, generator=g) * 10).to(dtype)
    b = (torch.randn(1000, generator=g) * 10).to(dtype)
    hi = torch.float64 if dtype == torch.float64 else torch.float32
    if dtype.is_floating_point:
        want = {"sum": a.to(hi) + b.to(hi), "max": torch.maximum(a.to(hi), b.to(hi)),
                "min": torch.minimum(a.to(hi), b.to(hi))}[op].to(dtype)
    else:
        want = {"sum": a + b, "max": torch.maximum(a, b), "min": torch.minimum(a, b)}[op]
    d = a.clone()
    assert native.utils.cpu_reduce(d.data_ptr(), b.data_ptr(), d.numel() * d.element_size(), name, op)
    assert torch.equal(d, want)


@pytest.mark.parametrize("bad", range(6))
def test_norm_kernels_refuse_addresses_off_the_16_byte_boundaries(native, bad):
    """The host refuses before anything is launched (there is no memory at these addresses)."""
    at = [4096 + 16 * i + (2 if i == bad else 0) for i in range(6)]
    with pytest.raises(RuntimeError, match="layernorm_fwd: invalid argument"):
        native.layernorm_fwd(*at, 0, 0, 4, 64, 1e-5, 0)
    if bad < 5:
        dy, x, g, dres, dx = at[:5]
        with pytest.raises(RuntimeError, match="layernorm_bwd: invalid argument"):
            native.layernorm_bwd(dy, x, g, 4096, 4096, dres, dx, 4096, 4096, 0, 4096, 4, 64, 0)



def test_layernorm_forward_forms(native):
    """One row per CTA (one barrier, as many CTAs as registers allow) where a CTA of several rows was slower; every form covers its row."""
    form = lambda rows, D: native.layernorm_fwd_form(rows, D, 148)  # noqa: E731   (warps, vectors, rows per CTA, one row by construction)
    for rows, D in ((1531, 2048), (600, 2048), (1000, 1536), (128, 1536), (1, 2560), (128, 4096), (1531, 3072), (3000, 2560), (4096, 5120), (600, 8192)):
        assert form(rows, D)[3], (rows, D)
    for rows, D in ((300, 2048), (444, 2048), (300, 4096), (2331, 2048), (16384, 2048), (1531, 768), (16384, 1024)):
        assert not form(rows, D)[3], (rows, D)
    for D in range(8, 8193, 8):
        for rows in (1, 148, 149, 444, 445, 888, 889, 1184, 1185, 1531, 4096, 70000):
            warps, vectors, per_cta, one_row = form(rows, D)
            assert warps * vectors * 32 >= D // 8 and 1 <= vectors <= 4 and 1 <= warps * per_cta <= 8 and (per_cta == 1 or not one_row), (rows, D)


def test_layernorm_backward_ring_is_for_many_rows(native):
    ring = lambda rows, D: native.layernorm_bwd_ring(rows, D, 148)  # noqa: E731
    assert not any(ring(1 << 20, D) for D in (8, 1024, 2048))
    assert not any(ring(rows, D) for rows, D in ((1, 2056), (600, 4096), (2368, 4096), (1, 8192), (600, 5120), (1036, 4104)))
    assert all(ring(rows, D) for rows, D in ((2369, 2056), (4096, 4096), (1037, 4104), (4096, 8192)))


@pytest.mark.parametrize("bucket", [False, True])
def test_embedding_backward_counts_negative_ids_from_the_end(bucket):
    """As its forward pass does, and as the fused token and position embedding does in both."""
    from pccl_b200.nn.linear import Embedding
    emb, V = Embedding(7, 8), 7
    ids = torch.tensor([[0, -1, 3], [-7, 6, -2]])
    if bucket:
        emb.weight.main_grad, emb.weight._pccl_written = torch.randn_like(emb.weight), False
    y = emb(ids)
    assert torch.equal(y, emb.weight[ids % V])
    dy = torch.randn(y.shape).bfloat16()
    y.backward(dy)
    want = torch.zeros_like(emb.weight).index_add_(0, ids.flatten() % V, dy.view(-1, 8))
    assert torch.equal(emb.weight.main_grad if bucket else emb.weight.grad, want)


def test_moe_gate_gradients_are_zeros_where_the_exchange_gives_up(native, monkeypatch):
    """Between ranks the kernel's entry barrier may run out, and then nothing is written."""
    from types import SimpleNamespace
    from pccl_b200.ops.moe import MoEExchange
    ex = MoEExchange.__new__(MoEExchange)
    ex.eng, ex.T, ex.K = SimpleNamespace(world=2), 64, 8
    monkeypatch.setattr(ex, "_exchange", lambda *a, **k: None, raising=False)
    made = []
    monkeypatch.setattr(torch, "empty", lambda *a, **k: made.append(a) or torch.full(*a, float("nan"), **k))
    assert torch.equal(ex.combine_dot(torch.zeros(64, 128), None, {"rows": None}), torch.zeros(64, 8))
    assert not made


def test_bucket_update_of_a_world_of_one_keeps_to_the_callers_blocks(native):
    plan = lambda count, blocks=0, threads=512: native.local_adamw_plan(count, blocks, threads, True, 148)  # noqa: E731   (CTAs of 128 threads, parameters)
    trip = 4 * 4 * 512                                         # parameters of a CTA in a launch: four trips of four warps
    assert plan(13 << 20) == (148, 148 * trip)
    assert plan(13 << 20, 8) == (32, 32 * trip) and plan(13 << 20, 1, 32) == (1, trip) and plan(13 << 20, 128) == (148, 148 * trip)
    big = 102_900_000
    assert plan(big) == (592, big) and plan(big, 8) == (32, big) and plan(big, 148) == (592, big)


def test_bucket_update_by_itself_is_one_launch(native):
    for count in (8, 5 << 20, 13 << 20, 102_900_000):
        assert native.local_adamw_plan(count, 0, 512, False, 148) == (592, count)
        assert native.local_adamw_plan(count, 4, 512, False, 148) == (16, count)


def test_moe_exchange_between_ranks_keeps_the_groups_that_were_measured(native):
    for dispatch, per_block in ((True, 6), (False, 4)):
        assert native.moe_group_threads(dispatch, 148 * per_block, 148, 1) == 64
        assert native.moe_group_threads(dispatch, 148 * per_block - 1, 148, 1) == 256
        assert all(native.moe_group_threads(dispatch, 1 << 20, blocks, world) == 256 for blocks in (1, 148) for world in (2, 4, 8))
