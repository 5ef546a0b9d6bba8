"""Tensor parallelism with sequence-parallel activations (Megatron's g / g-bar pair), every
collective fused into its GEMM kernel:

    forward   x_local --[all-gather -> GEMM]--> h = gelu(.) --[GEMM -> reduce-scatter]--> z_local
    backward  dz_local --[all-gather -> GEMM]--> dh ... --[GEMM -> reduce-scatter]--> dx_local

``ColumnParallelLinear`` holds W1[d_ff / TP, d_model], ``RowParallelLinear`` W2[d_model, d_ff / TP];
tokens (rows) are sharded over the ranks between the layers.  The backward GEMMs consume the weights
in transposed form through the kernels' MN-major operand path; weight gradients are local GEMMs on
the gathered activations that the forward kernels leave behind.
"""
from __future__ import annotations

import torch
import torch.nn as nn

from ..engine import Engine
from ..nn.linear import is_plain
from ..ops.fused_tp import AllGatherGemm, GemmReduceScatter
from ..ops.elementwise import colsum
from ..ops.gemm import gemm, gemm_dual


def _column_sums(dy: torch.Tensor) -> torch.Tensor:
    if dy.shape[1] % 8 == 0 and dy.data_ptr() % 16 == 0:
        return colsum(dy)
    return dy.sum(0, dtype=torch.float32).to(dy.dtype)


class _ColumnFn(torch.autograd.Function):
    @staticmethod
    def forward(ctx, x_local, weight, bias, layer):
        layer.ag.x_local.copy_(x_local)
        y = layer.ag(weight, bias)
        ctx.layer = layer
        ctx.save_for_backward(weight)
        ctx.has_bias = bias is not None
        return y

    @staticmethod
    def backward(ctx, dy):
        (weight,) = ctx.saved_tensors
        layer = ctx.layer
        dy = dy.contiguous()
        # dx_local = reduce_scatter_rows(dy @ W): W is [N1, K] = the [K_gemm, N_gemm] form -> w_t
        dx = layer.rs_bwd(dy, weight, w_t=True)
        dw = gemm(dy, layer.ag.x_full, a_t=True, b_t=True)            # [N1, K]
        return dx, dw, _column_sums(dy) if ctx.has_bias else None, None


class _RowFn(torch.autograd.Function):
    @staticmethod
    def forward(ctx, h, weight, bias, layer):
        z = layer.rs(h, weight, bias=bias)
        ctx.layer = layer
        ctx.save_for_backward(h, weight)
        ctx.has_bias = bias is not None
        return z

    @staticmethod
    def backward(ctx, dz_local):
        h, weight = ctx.saved_tensors
        layer = ctx.layer
        layer.ag_bwd.x_local.copy_(dz_local)
        dh = layer.ag_bwd(weight, w_t=True)                           # all_gather(dz) @ W2, W2 is [D, N1]
        dw = gemm(layer.ag_bwd.x_full, h, a_t=True, b_t=True)         # [D, N1]
        return dh, dw, _column_sums(dz_local.contiguous()) if ctx.has_bias else None, None


class _MlpFn(torch.autograd.Function):
    """Column-parallel layer, GELU and row-parallel layer as one node: GELU and its derivative run in the epilogues of the two
    all-gather GEMMs (the derivative's also sums the first layer's bias gradient), the second bias in the reduce-scatter's,
    and both weight gradients are one launch."""

    @staticmethod
    def forward(ctx, x_local, w1, b1, w2, b2, fc1, fc2):
        fc1.ag.x_local.copy_(x_local)
        act = torch.empty((fc1.ag.M, w1.shape[0]), dtype=torch.bfloat16, device=w1.device)
        pre = fc1.ag(w1, b1, gelu_out=act)
        z = fc2.rs(act, w2, bias=b2)
        ctx.save_for_backward(w1, w2, pre, act)
        ctx.layers, ctx.has_bias = (fc1, fc2), (b1 is not None, b2 is not None)
        return z

    @staticmethod
    def backward(ctx, dz_local):
        w1, w2, pre, act = ctx.saved_tensors
        fc1, fc2 = ctx.layers
        n1, d = w1.shape
        dz_local = dz_local.contiguous()
        fc2.ag_bwd.x_local.copy_(dz_local)
        sums = torch.empty(n1, dtype=torch.bfloat16, device=w1.device) if ctx.has_bias[0] else None
        dpre = fc2.ag_bwd(w2, w_t=True, dgelu=pre, colsum=sums)
        dx = fc1.rs_bwd(dpre, w1, w_t=True)
        dw1, dw2 = torch.empty_like(w1, memory_format=torch.contiguous_format), torch.empty_like(w2, memory_format=torch.contiguous_format)
        gemm_dual(dpre, fc1.ag.x_full, dw1, fc2.ag_bwd.x_full, act, dw2, a_t=True, b_t=True)
        return dx, dw1, sums, dw2, _column_sums(dz_local) if ctx.has_bias[1] else None, None, None


class ColumnParallelLinear(nn.Module):
    """y[tokens, out/TP] = all_gather_rows(x_local) @ W^T + b."""

    def __init__(self, eng: Engine, tokens: int, in_features: int, out_features: int, bias: bool = True, n_copy: int = 12,
                 init_std: float = 0.02):
        super().__init__()
        if out_features % eng.world:
            raise ValueError("ColumnParallelLinear: out_features must divide over the ranks")
        self.eng, self.tokens = eng, tokens
        n_local = out_features // eng.world
        self.weight = nn.Parameter(torch.empty((n_local, in_features), device="cuda", dtype=torch.bfloat16))
        nn.init.normal_(self.weight, std=init_std)
        self.bias = nn.Parameter(torch.zeros(n_local, device="cuda", dtype=torch.bfloat16)) if bias else None
        self.ag = AllGatherGemm(eng, tokens, in_features, n_copy=n_copy, flag_lane=4)
        self.rs_bwd = GemmReduceScatter(eng, tokens, in_features)

    def forward(self, x_local: torch.Tensor) -> torch.Tensor:
        return _ColumnFn.apply(x_local, self.weight, self.bias, self)


class RowParallelLinear(nn.Module):
    """z_local[tokens/TP, out] = reduce_scatter_rows(h @ W^T)  (+ b on every rank's rows)."""

    def __init__(self, eng: Engine, tokens: int, in_features: int, out_features: int, bias: bool = True, n_copy: int = 12,
                 init_std: float = 0.02):
        super().__init__()
        if in_features % eng.world:
            raise ValueError("RowParallelLinear: in_features must divide over the ranks")
        self.eng, self.tokens = eng, tokens
        k_local = in_features // eng.world
        self.weight = nn.Parameter(torch.empty((out_features, k_local), device="cuda", dtype=torch.bfloat16))
        nn.init.normal_(self.weight, std=init_std)
        self.bias = nn.Parameter(torch.zeros(out_features, device="cuda", dtype=torch.bfloat16)) if bias else None
        self.rs = GemmReduceScatter(eng, tokens, out_features)
        self.ag_bwd = AllGatherGemm(eng, tokens, out_features, n_copy=n_copy, flag_lane=6)

    def bias_in_epilogue(self) -> bool:
        """Whether the kernel can add the bias (its loads are 16 bytes of bf16); any other one is added by torch."""
        b = self.bias
        return b is None or (b.is_cuda and b.dtype == torch.bfloat16 and b.shape == self.weight.shape[:1] and b.is_contiguous() and b.data_ptr() % 16 == 0)

    def forward(self, h: torch.Tensor) -> torch.Tensor:
        if self.bias_in_epilogue():
            return _RowFn.apply(h, self.weight, self.bias, self)
        return _RowFn.apply(h, self.weight, None, self) + self.bias


class TensorParallelMLP(nn.Module):
    """x_local -> ColumnParallel -> GELU -> RowParallel -> z_local, rows sharded outside, d_ff sharded inside."""

    def __init__(self, eng: Engine, tokens: int, d_model: int, d_ff: int, n_copy: int = 12):
        super().__init__()
        self.fc1 = ColumnParallelLinear(eng, tokens, d_model, d_ff, n_copy=n_copy)
        self.fc2 = RowParallelLinear(eng, tokens, d_ff, d_model, n_copy=n_copy)

    def forward(self, x_local: torch.Tensor) -> torch.Tensor:
        fc1, fc2 = self.fc1, self.fc2
        # One node where both layers are this module's own with nobody listening in between, and the GELU-backward epilogue fits
        # (CTA pairs: 256 rows per rank; 32 columns).
        if (is_plain(fc1, ColumnParallelLinear) and is_plain(fc2, RowParallelLinear) and fc2.bias_in_epilogue()
                and (fc1.ag.M // fc1.eng.world) % 256 == 0 and fc1.weight.shape[0] % 32 == 0 and fc2.ag_bwd.ctas % 2 == 0):
            return _MlpFn.apply(x_local, fc1.weight, fc1.bias, fc2.weight, fc2.bias, fc1, fc2)
        return fc2(torch.nn.functional.gelu(fc1(x_local), approximate="tanh"))
