"""The two halves of a pre-norm transformer block around its attention as one autograd node and one native call each
(csrc/block_bindings.cc): residual sum, norm and QKV projection before it; projection, residual sum, norm and MLP behind it.

The kernels, their order and their results are those of ``LayerNorm.add_norm``, ``Linear`` and ``mlp`` called one by one; only the way
from one launch to the next is shorter, which is what a step of a small model consists of.  ``halves_apply`` says whether a block is
made of the layers that these halves stand for; any other block keeps the layers' own calls.
"""
from __future__ import annotations

from typing import Optional

import torch

from .._native import C
from ..ops.gemm import _PAIR_DEFAULT, _SKINNY_ROWS, _status_of, count_launch, records_graph, stream_handle
from .linear import Linear, LinearGelu, _as_operand, _deliver_bias, _finish_main_grad, _main_grad_out, _weight_grad, _weight_grad_pair, is_plain
from .norm import LayerNorm, _deliver, _grad_buffer, _rows, _writable

_bf16 = torch.bfloat16


def _form(rows: int) -> int:
    """The form that ``gemm`` takes for a product over ``rows`` rows."""
    if rows <= _SKINNY_ROWS:
        return C.GEMM_SKINNY
    return C.GEMM_PAIR if _PAIR_DEFAULT and rows > 128 else 0


def _fits(p: Optional[torch.Tensor], *shape: int) -> bool:
    return p is not None and p.dtype is _bf16 and p.shape == shape and p.is_cuda and p.is_contiguous() and p.data_ptr() % 16 == 0


def halves_apply(block, x: torch.Tensor) -> bool:
    """Whether the block's layers, as they are now, and its input are what the halves compute: the package's own layers without hooks
    or overrides, bf16 parameters of the block's shapes, an MLP width that the GELU-backward GEMM takes."""
    D = x.shape[-1]
    ln1, ln2, qkv, proj, fc1, fc2 = block.ln1, block.ln2, block.qkv, block.proj, block.fc1, block.fc2
    if not (is_plain(ln1, LayerNorm) and is_plain(ln2, LayerNorm) and is_plain(qkv, Linear) and is_plain(proj, Linear) and type(fc1) is LinearGelu
            and type(fc2) is Linear and "add_norm" not in ln1.__dict__ and "add_norm" not in ln2.__dict__):
        return False
    F = fc1.weight.shape[0]
    return (x.dtype is _bf16 and x.is_cuda and F % 32 == 0 and D % block.n_head == 0 and (D // block.n_head) % 8 == 0
            and _fits(ln1.weight, D) and _fits(ln1.bias, D) and _fits(ln2.weight, D) and _fits(ln2.bias, D)
            and _fits(qkv.weight, 3 * D, D) and _fits(qkv.bias, 3 * D) and _fits(proj.weight, D, D) and _fits(proj.bias, D)
            and _fits(fc1.weight, F, D) and _fits(fc1.bias, F) and _fits(fc2.weight, D, F) and _fits(fc2.bias, D))


def _attn_in_forward(x, delta, gamma, beta, w, bias, eps, want_stats):
    D = x.shape[-1]
    x2 = _rows(x, D)
    rows = x2.shape[0]
    s, d2 = x2, None
    if delta is not None:
        d2 = _rows(delta, D)
        s = torch.empty_like(x2)
    h = torch.empty_like(x2)
    qkv = x2.new_empty((rows, 3 * D))
    stats = x2.new_empty((2, rows), dtype=torch.float32) if want_stats else None
    C.block_attn_in(x2.data_ptr(), 0 if d2 is None else d2.data_ptr(), 0 if d2 is None else s.data_ptr(), gamma.data_ptr(), beta.data_ptr(), eps,
                    h.data_ptr(), 0 if stats is None else stats.data_ptr(), w.data_ptr(), bias.data_ptr(), qkv.data_ptr(), rows, D, _form(rows),
                    _status_of(x2), stream_handle())
    count_launch(2)
    return s, h, stats, qkv


def _split(qkv, B, T, heads):
    return tuple(t.transpose(1, 2) for t in qkv.view(B, T, 3, heads, -1).unbind(2))


class _AttnInFn(torch.autograd.Function):
    """(x, delta) -> (x + delta, q, k, v), without delta x -> (q, k, v); ``prev_bias`` is the bias of the layer that made delta, whose
    gradient the norm's backward yields (see ``LayerNorm.add_norm``)."""

    @staticmethod
    def forward(ctx, x, delta, gamma, beta, prev_bias, w, bias, heads, eps):
        B, T, D = x.shape
        s, h, stats, qkv = _attn_in_forward(x, delta, gamma, beta, w, bias, eps, True)
        ctx.save_for_backward(s, h, stats, gamma, w)
        ctx.params, ctx.prev_bias, ctx.bias = (gamma, beta), prev_bias, bias
        ctx.shape, ctx.heads, ctx.summed = x.shape, heads, delta is not None
        q, k, v = _split(qkv, B, T, heads)
        return (s.view(x.shape), q, k, v) if delta is not None else (q, k, v)

    @staticmethod
    def backward(ctx, *grads):
        s, h, stats, gamma, w = ctx.saved_tensors
        (B, T, D), heads, bias, rows = ctx.shape, ctx.heads, ctx.bias, s.shape[0]
        ds, grads = (grads[0], grads[1:]) if ctx.summed else (None, grads)
        gs = []
        for g in grads:
            g = g if g is not None else s.new_zeros((B, heads, T, D // heads))
            gs.append(g if g.stride(3) == 1 and not any(n % 8 for n in g.stride()[:3]) and g.data_ptr() % 16 == 0 else g.contiguous())
        dres = _rows(ds, D) if ds is not None else None
        dqkv = s.new_empty((rows, 3 * D))
        direct = _main_grad_out(bias, _bf16)
        db = direct if direct is not None else bias.new_empty(3 * D)
        dg, dbeta = (_grad_buffer(ctx, p) for p in ctx.params)
        dc = None
        if ctx.prev_bias is not None and ctx.needs_input_grad[4]:
            dc = _writable(ctx.prev_bias)
            dc = torch.empty_like(gamma) if dc is None else dc
        dh, dx = torch.empty_like(s), torch.empty_like(s)
        n_pack = C.colsum_parts(rows) * 3 * D
        parts = s.new_empty(n_pack + 3 * C.layernorm_bwd_parts(rows) * D, dtype=torch.float32)
        C.block_attn_in_bwd([g.data_ptr() for g in gs], [n for g in gs for n in g.stride()[:3]], dqkv.data_ptr(), B, T, heads, D // heads, db.data_ptr(),
                            parts.data_ptr(), w.data_ptr(), dh.data_ptr(), s.data_ptr(), gamma.data_ptr(), stats.data_ptr(),
                            0 if dres is None else dres.data_ptr(), dx.data_ptr(), dg.data_ptr(), dbeta.data_ptr(), 0 if dc is None else dc.data_ptr(),
                            parts.data_ptr() + 4 * n_pack, _form(rows), _status_of(s), stream_handle())
        count_launch(5)
        if direct is not None:
            _finish_main_grad(bias)
            db = None
        else:
            db = _deliver_bias(bias, db)
        dw = _weight_grad(dqkv, h, w)
        dxv = dx.view(ctx.shape)
        return dxv, (dxv if ctx.summed else None), dg, dbeta, (_deliver(ctx.prev_bias, dc) if dc is not None else None), dw, db, None, None


def _mlp_out_forward(a, x, wp, bp, gamma, beta, w1, b1, w2, b2, eps, for_backward):
    B, heads, T, hd = a.shape
    D, F = heads * hd, w1.shape[0]
    a2, x2 = _as_operand(a.transpose(1, 2).reshape(B * T, D)), _rows(x, D)
    rows = B * T
    d, s, h, out = torch.empty_like(x2), torch.empty_like(x2), torch.empty_like(x2), torch.empty_like(x2)
    act = x2.new_empty((rows, F))
    pre = torch.empty_like(act) if for_backward else None
    stats = x2.new_empty((2, rows), dtype=torch.float32) if for_backward else None
    C.block_mlp_out(a2.data_ptr(), a2.stride(0), wp.data_ptr(), bp.data_ptr(), d.data_ptr(), x2.data_ptr(), s.data_ptr(), gamma.data_ptr(), beta.data_ptr(),
                    eps, h.data_ptr(), 0 if stats is None else stats.data_ptr(), w1.data_ptr(), b1.data_ptr(), 0 if pre is None else pre.data_ptr(), act.data_ptr(), w2.data_ptr(),
                    b2.data_ptr(), out.data_ptr(), rows, D, F, _form(rows), _status_of(x2), stream_handle())
    count_launch(4)
    return a2, s, h, stats, pre, act, out


class _MlpOutFn(torch.autograd.Function):
    """(a, x) -> (s, out) with s = x + proj(a) and out = fc2(gelu(fc1(norm(s)))) for attention outputs a [B, heads, T, hd].  The bias
    gradient of fc2 is left to the norm that consumes ``out``."""

    @staticmethod
    def forward(ctx, a, x, wp, bp, gamma, beta, w1, b1, w2, b2, eps):
        a2, s, h, stats, pre, act, out = _mlp_out_forward(a, x, wp, bp, gamma, beta, w1, b1, w2, b2, eps, True)
        ctx.save_for_backward(a2, s, h, stats, pre, act, wp, gamma, w1, w2)
        ctx.params, ctx.proj_bias, ctx.fc1_bias, ctx.shape, ctx.a_shape = (gamma, beta), bp, b1, x.shape, a.shape
        return s.view(x.shape), out.view(x.shape)

    @staticmethod
    def backward(ctx, ds, dz):
        a2, s, h, stats, pre, act, wp, gamma, w1, w2 = ctx.saved_tensors
        rows, D = s.shape
        F = w1.shape[0]
        bp, b1 = ctx.proj_bias, ctx.fc1_bias
        dz2 = _as_operand(dz) if dz is not None else torch.zeros_like(s)
        dres = _rows(ds, D) if ds is not None else None
        direct = _main_grad_out(b1, _bf16)
        db1 = direct if direct is not None else b1.new_empty(F)
        dg, dbeta = (_grad_buffer(ctx, p) for p in ctx.params)
        dc = None
        if ctx.needs_input_grad[3]:
            dc = _writable(bp)
            dc = torch.empty_like(gamma) if dc is None else dc
        dpre = torch.empty_like(pre)
        dh, dx, da = torch.empty_like(s), torch.empty_like(s), torch.empty_like(s)
        n_sums = (rows + 31) // 32 * F
        parts = s.new_empty(n_sums + 3 * C.layernorm_bwd_parts(rows) * D, dtype=torch.float32)
        C.block_mlp_out_bwd(dz2.data_ptr(), dz2.stride(0), w2.data_ptr(), pre.data_ptr(), parts.data_ptr(), db1.data_ptr(), dpre.data_ptr(), w1.data_ptr(),
                            dh.data_ptr(), s.data_ptr(), gamma.data_ptr(), stats.data_ptr(), 0 if dres is None else dres.data_ptr(), dx.data_ptr(),
                            dg.data_ptr(), dbeta.data_ptr(), 0 if dc is None else dc.data_ptr(), parts.data_ptr() + 4 * n_sums, wp.data_ptr(),
                            da.data_ptr(), rows, D, F, _form(rows), _status_of(s), stream_handle())
        count_launch(6)
        if direct is not None:
            _finish_main_grad(b1)
            db1 = None
        else:
            db1 = _deliver_bias(b1, db1)
        dw1, dw2 = _weight_grad_pair(dpre, h, w1, dz2, act, w2)
        dbp = _deliver(bp, dc) if dc is not None else None
        dwp = _weight_grad(dx, a2, wp)
        B, heads, T, hd = ctx.a_shape
        return da.view(B, T, heads, hd).transpose(1, 2), dx.view(ctx.shape), dwp, dbp, dg, dbeta, dw1, db1, dw2, None, None


def attn_in(block, x, delta, prev_bias):
    """(residual stream, q, k, v) of a block for which ``halves_apply``; q, k, v are [B, heads, T, hd]."""
    ln, lin, heads = block.ln1, block.qkv, block.n_head
    if records_graph():
        got = _AttnInFn.apply(x, delta, ln.weight, ln.bias, prev_bias, lin.weight, lin.bias, heads, ln.eps)
        return got if delta is not None else (x,) + got
    B, T, _ = x.shape
    s, _, _, qkv = _attn_in_forward(x, delta, ln.weight, ln.bias, lin.weight, lin.bias, ln.eps, False)
    return (s.view(x.shape) if delta is not None else x,) + _split(qkv, B, T, heads)


def mlp_out(block, a, x):
    """(residual stream, output of the MLP) behind the attention output ``a`` [B, heads, T, hd] of such a block."""
    ln, args = block.ln2, (block.proj.weight, block.proj.bias, block.ln2.weight, block.ln2.bias, block.fc1.weight, block.fc1.bias, block.fc2.weight,
                           block.fc2.bias)
    if records_graph():
        return _MlpOutFn.apply(a, x, *args, ln.eps)
    _, s, _, _, _, _, out = _mlp_out_forward(a, x, *args, ln.eps, False)
    return s.view(x.shape), out.view(x.shape)
