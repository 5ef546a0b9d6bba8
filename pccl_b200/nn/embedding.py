"""Token and position embedding of a sequence model as one kernel per direction (csrc/kernels/elementwise.cu)."""
from __future__ import annotations

import torch

from .._native import C
from ..ops.gemm import count_launch, records_graph, stream_handle
from .linear import Embedding, _finish_main_grad, _grad_target, is_plain, row_indices
from .norm import _rows


def _forward(ids, tok, pos):
    B, T = ids.shape
    out = tok.new_empty((B, T, tok.shape[1]))
    C.embed_fwd(ids.data_ptr(), tok.data_ptr(), pos.data_ptr(), out.data_ptr(), B * T, T, tok.shape[0], tok.shape[1], stream_handle())
    count_launch()
    return out


class _TokenPositionFn(torch.autograd.Function):
    @staticmethod
    def forward(ctx, ids, tok, pos):
        ctx.save_for_backward(ids, tok, pos)
        return _forward(ids, tok, pos)

    @staticmethod
    def backward(ctx, dy):
        ids, tok, pos = ctx.saved_tensors
        B, T = ids.shape
        dy2 = _rows(dy, tok.shape[1])
        # the tables' gradients: the flat buckets' where a wrapper has attached them, and there behind what is in them already
        d_tok = _grad_target(tok) if ctx.needs_input_grad[1] else None
        d_pos = _grad_target(pos) if ctx.needs_input_grad[2] else None
        in_bucket = d_tok is not None, d_pos is not None
        if ctx.needs_input_grad[1]:
            if d_tok is None:
                d_tok = torch.zeros_like(tok)
            elif not getattr(tok, "_pccl_written", False):
                d_tok.zero_()
        add_pos = in_bucket[1] and bool(getattr(pos, "_pccl_written", False))
        if ctx.needs_input_grad[2]:
            if d_pos is None:
                d_pos = torch.empty_like(pos)
            if not add_pos and pos.shape[0] > T:
                d_pos[T:].zero_()
        # the kernel adds the tokens' rows in no fixed order; index_add_ honours torch.use_deterministic_algorithms
        by_kernel = d_tok
        if d_tok is not None and torch.are_deterministic_algorithms_enabled():
            d_tok.index_add_(0, row_indices(ids, tok.shape[0]), dy2)
            by_kernel = None
        if by_kernel is not None or d_pos is not None:
            C.embed_bwd(dy2.data_ptr(), ids.data_ptr(), 0 if by_kernel is None else by_kernel.data_ptr(), 0 if d_pos is None else d_pos.data_ptr(), B, T,
                        tok.shape[0], tok.shape[1], add_pos, stream_handle())
            count_launch()
        for there, p in zip(in_bucket, (tok, pos)):
            if there:
                _finish_main_grad(p)
        return None, (None if in_bucket[0] else d_tok), (None if in_bucket[1] else d_pos)


def _fits(p: torch.Tensor, D: int) -> bool:
    mg = _grad_target(p)
    return (p.dtype is torch.bfloat16 and p.is_cuda and p.dim() == 2 and p.shape[1] == D and p.is_contiguous() and p.data_ptr() % 16 == 0
            and (mg is None or (mg.dtype is torch.bfloat16 and mg.is_contiguous() and mg.data_ptr() % 16 == 0)))


# The backward walks the batch in one thread per eight columns of a position.  Up to 32 sequences it gains whatever their length.  Beyond that it
# depends on the positions as well: where they fill the device it would still gain (64 x 256 x 2048: 52 us against the layers' 294), where they are
# few it loses (64 x 1 x 256: 23.6 against 19.5; 1024 x 16 x 2048: 500 against 305).  The line is drawn by the batch alone, on the safe side.
_MAX_BATCH = 32


def _fused(ids: torch.Tensor, wte: torch.nn.Module, wpe: torch.nn.Module) -> bool:
    if not (is_plain(wte, Embedding) and is_plain(wpe, Embedding) and wte.weight is not wpe.weight):
        return False
    (B, T), D = ids.shape, wte.weight.shape[1]
    return (B <= _MAX_BATCH and ids.dtype is torch.int64 and ids.device == wte.weight.device == wpe.weight.device
            and 0 < ids.numel() * D < 1 << 34 and D % 8 == 0 and T <= wpe.weight.shape[0] and _fits(wte.weight, D) and _fits(wpe.weight, D))


def token_position(ids: torch.Tensor, wte: torch.nn.Module, wpe: torch.nn.Module) -> torch.Tensor:
    """``wte(ids) + wpe(arange(T))`` for ids [B, T].  Two plain ``Embedding`` layers with bf16 tables run as one kernel; anything else as
    the layers' own calls."""
    if _fused(ids, wte, wpe):
        ids = ids.contiguous()                # token windows are often slices of longer rows
        return _TokenPositionFn.apply(ids, wte.weight, wpe.weight) if records_graph() else _forward(ids, wte.weight, wpe.weight)
    return wte(ids) + wpe(torch.arange(ids.shape[1], device=ids.device))[None]
