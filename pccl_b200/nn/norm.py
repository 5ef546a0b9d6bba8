"""LayerNorm on this package's kernels (csrc/kernels/layernorm.cu): bf16 activations, fp32 statistics,
one pass over the activations per direction.  ``add_layer_norm`` is the residual connection of a pre-norm
transformer block and the norm that follows it as one kernel per direction."""
from __future__ import annotations

from typing import Optional, Tuple

import torch
import torch.nn as nn

from .._native import C
from ..ops.gemm import count_launch, records_graph, stream_handle


def _writable(param: Optional[torch.Tensor]) -> Optional[torch.Tensor]:
    """The flat-bucket gradient of ``param`` if the kernel may write it directly (nothing is in it yet this step)."""
    mg = getattr(param, "main_grad", None)
    if mg is None or mg.dtype != torch.bfloat16 or getattr(param, "_pccl_written", False) or not mg.is_contiguous() or mg.data_ptr() % 16:
        return None
    return mg


def _accumulates(ctx, param: torch.Tensor) -> bool:
    """Whether the running backward pass will accumulate a gradient of this node into ``param``: false for a frozen parameter and
    for an ``autograd.grad`` call, whether it asks for the parameter or for something else."""
    for node, _ in ctx.next_functions:
        if node is not None and getattr(node, "variable", None) is param:
            try:
                return torch._C._will_engine_execute_node(node)
            except RuntimeError:               # autograd.grad asked for this very leaf
                return False
    return False


def _grad_buffer(ctx, param: torch.Tensor) -> torch.Tensor:
    """Where a kernel puts the gradient of a parameter of the norm.  It always goes back to autograd, which knows who else
    contributes to it and which hooks see it; but where it will end in the flat bucket anyway it is written there to begin with,
    and the wrapper's hook finds nothing to copy.  The bucket is lent once per step: a second contribution gets memory of
    its own, and autograd adds the two.  Hooks other than the wrapper's may keep what they see: memory of its own as well."""
    mg, hooks = _writable(param), param._post_accumulate_grad_hooks
    if (mg is None or getattr(param, "_pccl_lent", True) or param._backward_hooks or (hooks is not None and len(hooks) > 1)
            or not _accumulates(ctx, param)):
        return torch.empty_like(param)
    param._pccl_lent = True
    return mg.view(mg.shape)                   # a tensor of its own: autograd keeps it as ``.grad`` without a copy


def _deliver(param: Optional[torch.Tensor], grad: torch.Tensor):
    """Hands a parameter's gradient to the data-parallel wrapper's flat bucket when there is one (and returns None),
    else returns it for autograd to accumulate."""
    if param is None:
        return None
    mg = getattr(param, "main_grad", None)
    if mg is None:
        return grad
    if grad is not mg:
        if getattr(param, "_pccl_written", False):
            mg.add_(grad.to(mg.dtype).view_as(mg))
        else:
            mg.copy_(grad.view_as(mg))
    param._pccl_written = True
    cb = getattr(param, "_pccl_ready", None)
    if cb is not None:
        cb()
    return None


def _ln_forward(x2, delta2, weight, bias, eps, want_stats=True):
    """(sum or None, y, fp32 [2, rows] with means and reciprocal deviations or None)"""
    rows, D = x2.shape
    y = torch.empty_like(x2)
    s = torch.empty_like(x2) if delta2 is not None else None
    stats = x2.new_empty((2, rows), dtype=torch.float32) if want_stats else None
    at = stats.data_ptr() if want_stats else 0
    C.layernorm_fwd(x2.data_ptr(), delta2.data_ptr() if delta2 is not None else 0, s.data_ptr() if s is not None else 0,
                    weight.data_ptr(), bias.data_ptr(), y.data_ptr(), at, at + 4 * rows if at else 0, rows, D, eps, stream_handle())
    count_launch()
    return s, y, stats


def _ln_backward(dy2, x2, weight, stats, dres2, dg, db, dc=None):
    """dx.  Writes the gradients of weight and bias to ``dg`` and ``db`` and, if given, the column sums of dx to ``dc``."""
    rows, D = x2.shape
    dx = torch.empty_like(x2)
    partials = x2.new_empty(3 * C.layernorm_bwd_parts(rows) * D, dtype=torch.float32)
    at = stats.data_ptr()
    C.layernorm_bwd(dy2.data_ptr(), x2.data_ptr(), weight.data_ptr(), at, at + 4 * rows,
                    dres2.data_ptr() if dres2 is not None else 0, dx.data_ptr(), dg.data_ptr(), db.data_ptr(),
                    dc.data_ptr() if dc is not None else 0, partials.data_ptr(), rows, D, stream_handle())
    count_launch(2)
    return dx


def _rows(t: torch.Tensor, D: int) -> torch.Tensor:
    """``t`` as contiguous rows on a 16-byte boundary, as the kernels read them."""
    t2 = t.reshape(-1, D)
    if not t2.is_contiguous():
        return t2.contiguous()
    return t2 if t2.data_ptr() % 16 == 0 else t2.clone()


class _LayerNormFn(torch.autograd.Function):
    @staticmethod
    def forward(ctx, x, weight, bias, eps):
        x2 = _rows(x, x.shape[-1])
        _, y, stats = _ln_forward(x2, None, weight, bias, eps)
        ctx.save_for_backward(x2, weight, stats)
        ctx.params = (weight, bias)
        ctx.shape = x.shape
        return y.view(x.shape)

    @staticmethod
    def backward(ctx, dy):
        x2, weight, stats = ctx.saved_tensors
        dg, db = (_grad_buffer(ctx, p) for p in ctx.params)
        dx = _ln_backward(_rows(dy, x2.shape[1]), x2, weight, stats, None, dg, db)
        return dx.view(ctx.shape), dg, db, None


class _AddLayerNormFn(torch.autograd.Function):
    """(x, delta) -> (s, y) with s = x + delta and y = LayerNorm(s).  ``prev_bias`` is the bias of the linear layer that
    produced ``delta`` (or None): the gradient of ``delta`` summed over rows is that bias's gradient, and backward computes
    it while it has the rows in registers, so that layer does not make a pass of its own for it."""

    @staticmethod
    def forward(ctx, x, delta, weight, bias, prev_bias, eps):
        D = x.shape[-1]
        x2, d2 = _rows(x, D), _rows(delta, D)
        s, y, stats = _ln_forward(x2, d2, weight, bias, eps)
        ctx.save_for_backward(s, weight, stats)
        ctx.params, ctx.prev_bias = (weight, bias), prev_bias
        ctx.shape = x.shape
        return s.view(x.shape), y.view(x.shape)

    @staticmethod
    def backward(ctx, ds, dy):
        s, weight, stats = ctx.saved_tensors
        D = s.shape[1]
        if dy is None:
            dy = torch.zeros_like(s)
        dres = _rows(ds, D) if ds is not None else None
        want = ctx.prev_bias is not None and ctx.needs_input_grad[4]
        dg, db = (_grad_buffer(ctx, p) for p in ctx.params)
        dc = None
        if want:
            dc = _writable(ctx.prev_bias)
            dc = torch.empty_like(weight) if dc is None else dc
        dx = _ln_backward(_rows(dy, D), s, weight, stats, dres, dg, db, dc)
        dxv = dx.view(ctx.shape)
        return dxv, dxv, dg, db, (_deliver(ctx.prev_bias, dc) if want else None), None


class LayerNorm(nn.Module):
    def __init__(self, dim: int, eps: float = 1e-5, device=None, dtype=torch.bfloat16):
        super().__init__()
        if dim % 8 or dim > 8192 or dtype != torch.bfloat16:
            raise ValueError("LayerNorm: bf16, dim % 8 == 0 and dim <= 8192")
        self.eps = eps
        self.weight = nn.Parameter(torch.ones(dim, device=device, dtype=dtype))
        self.bias = nn.Parameter(torch.zeros(dim, device=device, dtype=dtype))

    def forward(self, x: torch.Tensor) -> torch.Tensor:
        weight, bias = self.weight, self.bias
        if records_graph():
            return _LayerNormFn.apply(x, weight, bias, self.eps)
        return _ln_forward(_rows(x, x.shape[-1]), None, weight, bias, self.eps, False)[1].view(x.shape)

    def add_norm(self, x: torch.Tensor, delta: torch.Tensor, prev_bias: Optional[torch.Tensor] = None) -> Tuple[torch.Tensor, torch.Tensor]:
        """Returns ``(x + delta, LayerNorm(x + delta))``.  Pass the bias of the linear layer that produced ``delta`` as
        ``prev_bias`` when that layer was told to leave its bias gradient to this norm (``Linear(..., defer_bias_grad=True)``)."""
        weight, bias = self.weight, self.bias
        if records_graph():
            return _AddLayerNormFn.apply(x, delta, weight, bias, prev_bias, self.eps)
        D = x.shape[-1]
        s, y, _ = _ln_forward(_rows(x, D), _rows(delta, D), weight, bias, self.eps, False)
        return s.view(x.shape), y.view(x.shape)
