"""What a user of this package has one GPU do, as cases for timing: training steps and inference of the GPT model, linear
layers by themselves, a tensor-parallel MLP's share of one rank, block-scaled fp8 MLPs, and mixture-of-experts layers --
each from the smallest call in use to the largest, with odd sizes in between.

``listed()`` names the cases, ``draw(rng)`` gives another one of the same ranges, ``prepare`` makes what a program has in
hand before the call, ``run`` is one pass through the public entry points, ``work`` the bytes and operations that the pass
cannot do without, and ``tolerance`` how far two correct implementations may lie apart.
"""
from __future__ import annotations

import gc
import math

import torch

from pccl_b200.engine import Engine
from pccl_b200.models.gpt import GPT, GPTConfig
from pccl_b200.nn.linear import Linear
from pccl_b200.ops.gemm import gemm_fp8, gemm_mx8, quant_blocks, quant_blocks_mx, quant_rows, quant_rows_mx
from pccl_b200.parallel.dp import ShardedDataParallel
from pccl_b200.parallel.ep import MoELayer
from pccl_b200.parallel.tp import TensorParallelMLP


def listed():
    return [
        # The configuration of the smoke test and of the CPU-sized examples: a step is some eighty launches of a few
        # microseconds each, so what counts is latency, launches and host work.
        {"name": "train_tiny", "kind": "train", "layers": 2, "d": 256, "heads": 4, "vocab": 1001, "batch": 2, "seq": 128},
        # A small model on a batch whose row count fits no tile (777 positions, 3 sequences), heads of 64, full vocabulary.
        {"name": "train_ragged", "kind": "train", "layers": 4, "d": 768, "heads": 12, "vocab": 50257, "batch": 3, "seq": 777},
        # The benchmark of the repository: GPT-1.3B, 8 sequences of 2048 tokens per GPU, bf16, AdamW.
        {"name": "train_1p3b", "kind": "train", "layers": 24, "d": 2048, "heads": 16, "vocab": 50257, "batch": 8, "seq": 2048},
        # Evaluation (prefill) with the same model: the logits of one sequence of odd length, no gradients.
        {"name": "logits_1p3b", "kind": "logits", "layers": 24, "d": 2048, "heads": 16, "vocab": 50257, "batch": 1, "seq": 1531},
        # One linear layer at the token counts of decoding: the weights are read once for a handful of rows.
        {"name": "linear_decode", "kind": "linear", "rows": 24, "n_in": 8192, "n_out": 8192},
        # Forward and backward of one linear layer with sizes that are multiples of 8 and of nothing else.
        {"name": "linear_ragged", "kind": "linear_train", "rows": 1999, "n_in": 1416, "n_out": 3000},
        # One rank's share of the tensor-parallel MLP benchmark (8192 tokens, 8192 -> 28672 / 8 -> 8192), forward and backward,
        # through the fused all-gather -> GEMM and GEMM -> reduce-scatter kernels in a world of one.
        {"name": "tp_mlp", "kind": "tp_mlp", "tokens": 8192, "d": 8192, "d_ff": 3584},
        # The same share in block-scaled fp8 (1 x 128 activation scales, 128 x 128 weight scales, fp32 scales), inference.
        {"name": "mlp_fp8", "kind": "mlp_fp8", "tokens": 8192, "d": 8192, "d_ff": 3584},
        # Block-scaled fp8 with power-of-two scales that the tensor core applies, on an odd number of tokens.
        {"name": "mlp_mx8", "kind": "mlp_mx8", "tokens": 1531, "d": 8192, "d_ff": 3584},
        # One rank's share of the mixture-of-experts benchmark (32 experts, 4096 tokens, top-8), inference ...
        {"name": "moe_serve", "kind": "moe_serve", "tokens": 4096, "hidden": 7168, "d_ff": 2048, "experts": 32, "topk": 8},
        # ... the same layer at the token count of decoding, where the experts' weights are what is read ...
        {"name": "moe_decode", "kind": "moe_serve", "tokens": 64, "hidden": 7168, "d_ff": 2048, "experts": 32, "topk": 8},
        # ... and training of a smaller layer on an odd number of tokens.
        {"name": "moe_train", "kind": "moe_train", "tokens": 2001, "hidden": 2048, "d_ff": 1024, "experts": 32, "topk": 4},
    ]


def _log_int(rng, lo, hi, step=1):
    """An integer between lo and hi, spread over its logarithm, rounded to a multiple of ``step``."""
    v = math.exp(rng.uniform(math.log(lo), math.log(hi)))
    return max(step, int(v / step + 0.5) * step)


def draw(rng):
    kind = rng.choice(["train", "train", "logits", "linear", "linear_train", "tp_mlp", "mlp_fp8", "mlp_mx8", "moe_serve", "moe_serve", "moe_train"])
    if kind in ("train", "logits"):
        head_dim = rng.choice([64, 128])
        d = head_dim * _log_int(rng, 256 // head_dim, 2048 // head_dim)
        vocab = rng.choice([1001, 8191, 32000, 50257])
        layers = rng.randint(2, 24)
        top = 16384 if kind == "train" else 4096
        seq = _log_int(rng, 96, 2048)
        batch = max(1, min(16, _log_int(rng, 128, top) // seq))
        return {"kind": kind, "layers": layers, "d": d, "heads": d // head_dim, "vocab": vocab, "batch": batch, "seq": seq}
    if kind == "linear":
        return {"kind": kind, "rows": _log_int(rng, 1, 8192), "n_in": _log_int(rng, 512, 8192, 8), "n_out": _log_int(rng, 512, 8192, 8)}
    if kind == "linear_train":
        return {"kind": kind, "rows": _log_int(rng, 64, 16384), "n_in": _log_int(rng, 256, 8192, 8), "n_out": _log_int(rng, 256, 8192, 8)}
    if kind == "tp_mlp":
        return {"kind": kind, "tokens": _log_int(rng, 128, 8192, 128), "d": _log_int(rng, 1024, 8192, 256), "d_ff": _log_int(rng, 1024, 8192, 128)}
    if kind in ("mlp_fp8", "mlp_mx8"):
        return {"kind": kind, "tokens": _log_int(rng, 16, 16384), "d": _log_int(rng, 1024, 8192, 128), "d_ff": _log_int(rng, 1024, 8192, 128)}
    experts = rng.choice([8, 16, 32])
    if kind == "moe_serve":
        return {"kind": kind, "tokens": _log_int(rng, 16, 4096), "hidden": _log_int(rng, 1024, 7168, 128), "d_ff": _log_int(rng, 512, 2048, 128),
                "experts": experts, "topk": rng.choice([2, 4, 8])}
    return {"kind": kind, "tokens": _log_int(rng, 128, 4096), "hidden": _log_int(rng, 1024, 4096, 128), "d_ff": _log_int(rng, 512, 2048, 128),
            "experts": experts, "topk": rng.choice([2, 4, 8])}


WORKSPACE = 512 << 20                      # the engine's own part of the heap (256 MiB by default) and room for alignment


# ---- states ------------------------------------------------------------------------------------------------------------
def _randn(shape, scale=1.0, dtype=torch.bfloat16):
    return (torch.randn(shape, device="cuda", dtype=torch.float32) * scale).to(dtype)


def _moe_engine(case):
    """A world of one whose symmetric heap holds the exchange buffers of the layer (rows of e4m3, bf16 and bf16)."""
    cap = 2 * case["tokens"] * case["topk"] + 256
    heap = cap * (case["hidden"] * 5 + case["hidden"] // 32 + 256) + WORKSPACE
    eng = Engine(0, 1)
    eng.initEngine("cuda", heap)
    return eng


def prepare(case, seed):
    kind = case["kind"]
    if kind == "train":
        torch.cuda.synchronize()          # a wrapper and its parameters hold one another: give an earlier state's memory back,
        gc.collect()                      # once nothing in flight uses it
        torch.cuda.empty_cache()
    torch.manual_seed(seed)
    if kind in ("train", "logits"):
        cfg = GPTConfig(n_layer=case["layers"], n_head=case["heads"], d_model=case["d"], seq_len=case["seq"], vocab_size=case["vocab"])
        model = GPT(cfg, device="cuda")
        ids = torch.randint(0, case["vocab"], (case["batch"], case["seq"]), device="cuda")
        if kind == "logits":
            return {"kind": kind, "model": model, "ids": ids}
        dp = ShardedDataParallel(model)
        return {"kind": kind, "dp": dp, "ids": ids, "targets": ids.roll(-1, 1)}
    if kind in ("linear", "linear_train"):
        layer = Linear(case["n_in"], case["n_out"], device="cuda")
        layer.bias.data.copy_(_randn(case["n_out"], 0.1))
        st = {"kind": kind, "layer": layer, "x": _randn((case["rows"], case["n_in"]))}
        if kind == "linear_train":
            st["x"].requires_grad_(True)
            st["dy"] = _randn((case["rows"], case["n_out"]))
        return st
    if kind == "tp_mlp":
        eng = Engine(0, 1)
        eng.initEngine("cuda", 6 * case["tokens"] * case["d"] * 2 + 4 * case["tokens"] * case["d_ff"] + WORKSPACE)
        layer = TensorParallelMLP(eng, case["tokens"], case["d"], case["d_ff"])
        x = _randn((case["tokens"], case["d"])).requires_grad_(True)
        return {"kind": kind, "engine": eng, "layer": layer, "params": list(layer.parameters()), "x": x, "dz": _randn((case["tokens"], case["d"]))}
    if kind in ("mlp_fp8", "mlp_mx8"):
        qb = quant_blocks if kind == "mlp_fp8" else quant_blocks_mx
        return {"kind": kind, "x": _randn((case["tokens"], case["d"])), "w1": qb(_randn((case["d_ff"], case["d"]), 0.02)),
                "b1": _randn(case["d_ff"], 0.1), "w2": qb(_randn((case["d"], case["d_ff"]), 0.02)), "b2": _randn(case["d"], 0.1)}
    eng = _moe_engine(case)
    layer = MoELayer(eng, case["tokens"], case["hidden"], case["d_ff"], case["experts"], case["topk"])
    x = _randn((case["tokens"], case["hidden"]))
    gate_logits = torch.randn((case["tokens"], case["experts"]), device="cuda")
    st = {"kind": kind, "engine": eng, "layer": layer, "x": x, "gate_logits": gate_logits}
    if kind == "moe_train":
        x.requires_grad_(True)
        gate_logits.requires_grad_(True)
        st["dout"] = _randn((case["tokens"], case["hidden"]))
    return st


def run(state):
    kind = state["kind"]
    if kind == "train":
        # forward, backward with the gradient buckets' reduce-scatter + AdamW on the side stream, the updated parameters
        dp = state["dp"]
        loss = dp.train_step(state["ids"], state["targets"])
        return {"loss": loss, "grads": dp.flat_grads, "params": dp.flat_params}
    if kind == "logits":
        with torch.no_grad():
            return state["model"].logits(state["ids"])
    if kind == "linear":
        with torch.no_grad():
            return state["layer"](state["x"])
    if kind == "linear_train":
        layer = state["layer"]
        y = layer(state["x"])
        dx, dw, db = torch.autograd.grad(y, [state["x"], layer.weight, layer.bias], state["dy"])
        return {"y": y, "dx": dx, "dw": dw, "db": db}
    if kind == "tp_mlp":
        z = state["layer"](state["x"])
        return {"z": z, "grads": torch.autograd.grad(z, [state["x"]] + state["params"], state["dz"])}
    if kind == "mlp_fp8":
        h = gemm_fp8(*quant_rows(state["x"]), *state["w1"], bias=state["b1"], gelu_inplace=True)
        return gemm_fp8(*quant_rows(h), *state["w2"], bias=state["b2"])
    if kind == "mlp_mx8":
        h = gemm_mx8(*quant_rows_mx(state["x"]), *state["w1"], bias=state["b1"], gelu_inplace=True)
        return gemm_mx8(*quant_rows_mx(h), *state["w2"], bias=state["b2"])
    layer = state["layer"]
    if kind == "moe_serve":
        with torch.no_grad():
            return layer(state["x"], state["gate_logits"])
    out = layer(state["x"], state["gate_logits"])
    grads = torch.autograd.grad(out, [state["x"], state["gate_logits"], layer.w1, layer.w2], state["dout"])
    return {"out": out, "grads": grads}


# ---- what a pass cannot do without ----------------------------------------------------------------------------------------
def work(case):
    kind = case["kind"]
    if kind in ("train", "logits"):
        L, d, V, T, S = case["layers"], case["d"], case["vocab"], case["batch"] * case["seq"], case["seq"]
        mats = L * 12 * d * d
        params = mats + L * 13 * d + V * d + S * d + 2 * d
        fwd = 2.0 * T * (mats + V * d) + L * 2.0 * T * S * d          # causal attention: half of the S x S products, twice
        if kind == "logits":
            return {"bytes": 2.0 * params + 8.0 * T + 2.0 * T * V, "flops": fwd}
        # parameters read and written (bf16), gradients written, fp32 master and both moments read and written
        return {"bytes": params * (2 + 2 + 2 + 24.0) + 16.0 * T, "flops": 3 * fwd}
    if kind in ("linear", "linear_train"):
        M, K, N = case["rows"], case["n_in"], case["n_out"]
        if kind == "linear":
            return {"bytes": 2.0 * (M * K + N * K + N + M * N), "flops": 2.0 * M * N * K}
        return {"bytes": 2.0 * (M * K + N * K + N + M * N) + 2.0 * (M * N + M * K + N * K + N), "flops": 6.0 * M * N * K}
    if kind == "tp_mlp":
        M, D, F = case["tokens"], case["d"], case["d_ff"]
        return {"bytes": 2.0 * (4 * M * D + 2 * (2 * D * F + F + D)), "flops": 12.0 * M * D * F}
    if kind in ("mlp_fp8", "mlp_mx8"):
        M, D, F = case["tokens"], case["d"], case["d_ff"]
        # e4m3 products run at twice the bf16 rate: counted as they are
        return {"bytes": 4.0 * M * D + 2.0 * D * F + 2.0 * (D + F), "flops": 4.0 * M * D * F}
    M, H, F, E, k = case["tokens"], case["hidden"], case["d_ff"], case["experts"], case["topk"]
    used = E * (1.0 - (1.0 - k / E) ** M)                              # experts that some token is routed to
    weights = 2.0 * 2 * used * H * F
    if kind == "moe_serve":
        return {"bytes": weights + 4.0 * M * H + 4.0 * M * E, "flops": 4.0 * M * k * H * F}
    return {"bytes": weights + 2.0 * 2 * E * H * F + 8.0 * M * H + 8.0 * M * E, "flops": 12.0 * M * k * H * F}


def tolerance(case):
    return TOLERANCE[case["kind"]]


# About four times what was measured between two implementations of the same precision: the training step with its fused
# against its unfused blocks (gradients 0.4 to 0.9 % apart in norm, single elements by up to their size: a gradient of a
# rare token is a sum of few bf16 terms), the model's logits with its GEMMs against fp32 matrix products (1.4 %), the other
# paths against fp32 or another order of sums (0.17 % is the rounding of a bf16 result; 0.4 % for the two combine forms).
TOLERANCE = {
    "train": {"rel": 0.03, "max": 0.99},
    "logits": {"rel": 0.03, "max": 0.32},
    "linear": {"rel": 7e-3, "max": 0.016},
    "linear_train": {"rel": 7e-3, "max": 0.016},
    "tp_mlp": {"rel": 7e-3, "max": 0.032},
    "mlp_fp8": {"rel": 7e-3, "max": 0.12},
    "mlp_mx8": {"rel": 7e-3, "max": 0.06},
    "moe_serve": {"rel": 0.016, "max": 0.13},
    "moe_train": {"rel": 7e-3, "max": 0.1},
}
