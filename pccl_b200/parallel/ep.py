"""Expert parallelism: a mixture-of-experts feed-forward layer whose token exchange runs on this
library's dispatch / combine kernels (fp8 payload with per-128 scales out, gate-weighted bf16 back)
and whose experts run as one grouped tcgen05 GEMM per projection.

The layer trains: its backward pass reuses the same exchange.  The gradient of the output goes to the
experts' ranks through the dispatch kernel, weighted by the gate probability of each assignment (the
e4m3 payload of a row is the same for all of its destinations, only the block scales are multiplied);
the experts' input gradients come back through the combine kernel; the gradients of the gate weights
are dot products of the upstream gradient with the expert output rows, taken by a third kernel that
pulls the rows like the combine does.  The expert GEMMs of the backward pass are the grouped kernel
again (input gradients, on the weights as they are stored) and one launch for the weight gradients of all
experts, whose reduction dimension is the expert's row count.  No step waits for the host.  The reference has no model code; this is the EP strategy it names.
"""
from __future__ import annotations

import torch
import torch.nn as nn

from ..engine import Engine
from ..ops.moe import MoEExchange, grouped_gemm, grouped_wgrad


class _MoEFn(torch.autograd.Function):
    """out[t] = sum_k p[t,k] * W2_e gelu(W1_e x[t]) over the top-k experts e of token t.  One forward per backward:
    the expert outputs stay in the exchange's symmetric buffer until the backward pass has read them."""

    @staticmethod
    def forward(ctx, x, gate_logits, w1, w2, ex: MoEExchange):
        ids, probs, plan = ex.route_and_plan(gate_logits)
        xr = ex.deliver(x, ids, plan)                            # what the experts see (after the e4m3 round trip)
        d_ff = w1.shape[0] // ex.epr
        h = torch.empty((xr.shape[0], d_ff), dtype=torch.bfloat16, device=xr.device)
        h_pre = grouped_gemm(xr, w1, plan["row_off"], d_ff, gelu_out=h)
        grouped_gemm(h, w2, plan["row_off"], ex.H, out=ex.y)
        out = ex.combine(ids, probs, plan)
        ctx.save_for_backward(gate_logits, w1, w2, ids, probs, plan["rows"], plan["row_off"], plan["n_rows"], xr, h_pre, h)
        ctx.ex = ex
        return out

    @staticmethod
    def backward(ctx, dout):
        gate_logits, w1, w2, ids, probs, rows, row_off, n_rows, xr, h_pre, h = ctx.saved_tensors
        ex = ctx.ex
        plan = {"rows": rows, "row_off": row_off, "n_rows": n_rows}
        epr, H = ex.epr, ex.H
        d_ff = w1.shape[0] // epr
        dout = dout.contiguous()
        # gate weights: d p[t,k] = <dout[t], expert output row>, while the forward outputs are still in ex.y
        dp = ex.combine_dot(dout, ids, plan)
        # output gradients to the experts, each weighted by its gate probability
        g = ex.deliver(dout, ids, plan, probs=probs)
        # experts: the same grouped kernel on the weights as they lie, gelu' in its epilogue, then all weight gradients at once
        dh_pre = grouped_gemm(g, w2, row_off, d_ff, b_t=True, dgelu=h_pre)
        grouped_gemm(dh_pre, w1, row_off, H, b_t=True, out=ex.y)
        dw1, dw2 = grouped_wgrad(dh_pre, xr, g, h, row_off)
        # input gradients back to the tokens: a plain sum over the k assignments (the gate weight went out with dout)
        dx = ex.combine(ids, None, plan)
        dlogits = ex.route_backward(gate_logits, ids, dp)
        return dx, dlogits.to(gate_logits.dtype), dw1, dw2, None


class MoELayer(nn.Module):
    def __init__(self, eng: Engine, tokens: int, d_model: int, d_ff: int, n_experts: int, topk: int = 8,
                 capacity_factor: float = 2.0, init_std: float = 0.02):
        super().__init__()
        self.eng, self.topk = eng, topk
        epr = n_experts // eng.world
        self.gate = nn.Parameter(torch.randn(n_experts, d_model, device="cuda", dtype=torch.bfloat16) * init_std)
        self.w1 = nn.Parameter(torch.randn(epr * d_ff, d_model, device="cuda", dtype=torch.bfloat16) * init_std)
        self.w2 = nn.Parameter(torch.randn(epr * d_model, d_ff, device="cuda", dtype=torch.bfloat16) * init_std)
        self.exchange = MoEExchange(eng, tokens, d_model, n_experts, topk, capacity_factor)

    def forward(self, x: torch.Tensor, gate_logits: torch.Tensor = None) -> torch.Tensor:
        """With gradients enabled the layer runs as an autograd node (see ``_MoEFn``); under ``torch.no_grad()`` it takes
        the serving path, which fuses the GELU into the first grouped GEMM and keeps nothing for a backward pass."""
        if gate_logits is None:
            gate_logits = (x @ self.gate.t()).float()
        if torch.is_grad_enabled() and (x.requires_grad or gate_logits.requires_grad or self.w1.requires_grad):
            return _MoEFn.apply(x, gate_logits, self.w1, self.w2, self.exchange)
        with torch.no_grad():
            return self.exchange.forward(x, gate_logits, self.w1, self.w2)
