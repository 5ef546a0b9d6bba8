"""Expert-parallel MoE: routing plan, fp8 dispatch, grouped expert FFN, weighted combine
(csrc/kernels/moe.cu).  Everything stays on the device: token counts per expert are exchanged with
this library's all-gather and turned into receive offsets with a few tensor ops, and the grouped
GEMM reads the per-expert row ranges from device memory, so no step needs the host to know sizes.
"""
from __future__ import annotations

import weakref
from typing import Dict, Optional, Tuple

import torch

from .._native import C
from ..engine import Engine
from . import collectives as coll
from .gemm import count_launch, status_words, stream_handle


def quant_fp8_rows(x: torch.Tensor) -> Tuple[torch.Tensor, torch.Tensor]:
    """bf16 [rows, hidden] -> (e4m3 bytes [rows, hidden], fp32 scales [rows, hidden/128]); 1 x 128 blocks."""
    rows, hidden = x.shape
    q = torch.empty((rows, hidden), dtype=torch.uint8, device=x.device)
    s = torch.empty((rows, hidden // 128), dtype=torch.float32, device=x.device)
    C.quant_fp8_rows(x.data_ptr(), q.data_ptr(), s.data_ptr(), rows, hidden, stream_handle())
    count_launch()
    return q, s


def quant_fp8_blocks(w: torch.Tensor) -> Tuple[torch.Tensor, torch.Tensor]:
    """bf16 [rows, cols] weights -> (e4m3 bytes, fp32 scales [rows/128, cols/128]); 128 x 128 blocks."""
    rows, cols = w.shape
    q = torch.empty((rows, cols), dtype=torch.uint8, device=w.device)
    s = torch.empty((rows // 128, cols // 128), dtype=torch.float32, device=w.device)
    C.quant_fp8_blocks(w.data_ptr(), q.data_ptr(), s.data_ptr(), rows, cols, stream_handle())
    count_launch()
    return q, s


def grouped_gemm(a: torch.Tensor, b: torch.Tensor, row_off: torch.Tensor, n: int, out: Optional[torch.Tensor] = None,
                 gelu: bool = False, *, b_t: bool = False, gelu_out: Optional[torch.Tensor] = None,
                 dgelu: Optional[torch.Tensor] = None) -> torch.Tensor:
    """Rows [row_off[g], row_off[g+1]) of ``a`` [*, K] times ``b[g*n:(g+1)*n]`` ([groups*n, K]) ^T -> same rows of out [*, n].
    ``b_t``: the blocks of ``b`` are [K, n] (stacked [groups*K, n]) and not transposed.  ``gelu_out`` receives gelu_tanh(out);
    ``dgelu`` (a pre-activation) makes it ``out = product * gelu_tanh'(dgelu)``; both have ``out``'s shape and strides."""
    groups, K = row_off.numel() - 1, a.shape[1]
    if b_t and K % 64:                 # the kernel reads k in blocks of 64, which must not reach into the next group's weights
        b, b_t = b.view(groups, K, n).transpose(1, 2).reshape(groups * n, K), False
    if out is None:
        out = torch.empty((a.shape[0], n), dtype=torch.bfloat16, device=a.device)
    side = gelu_out if gelu_out is not None else dgelu
    if side is not None and ((gelu_out is not None and dgelu is not None) or gelu or side.dtype != torch.bfloat16 or side.shape != out.shape
                             or side.stride() != out.stride()):
        raise ValueError("grouped_gemm: one of gelu, gelu_out and dgelu, a bf16 tensor of out's shape and strides")
    flags = (C.GEMM_GELU_INPLACE if gelu else 0) | (C.GEMM_B_MN if b_t else 0)
    if side is not None:
        flags |= C.GEMM_GELU if gelu_out is not None else C.GEMM_DGELU
    C.gemm_grouped(a.data_ptr(), a.stride(0), b.data_ptr(), b.stride(0), out.data_ptr(), out.stride(0), row_off.data_ptr(), groups,
                   a.shape[0], n, K, flags, 0, status_words().data_ptr(), stream_handle(),
                   side.data_ptr() if side is not None else 0)
    count_launch()
    return out


def grouped_wgrad(a0: torch.Tensor, b0: torch.Tensor, a1: torch.Tensor, b1: torch.Tensor, row_off: torch.Tensor) -> Tuple[torch.Tensor, torch.Tensor]:
    """``d_q[g] = a_q[rows of g]^T @ b_q[rows of g]`` for q = 0, 1 and every group, as [groups * M_q, N_q] (zeros for a group
    without rows); a_q [rows, M_q] and b_q [rows, N_q] are bf16 over the same rows."""
    groups, rows = row_off.numel() - 1, a0.shape[0]
    problems, outs = [], []
    for a, b in ((a0, b0), (a1, b1)):
        if a.shape[0] != rows or b.shape[0] != rows or a.stride(1) != 1 or b.stride(1) != 1:
            raise ValueError("grouped_wgrad: operands must be row-major over the same rows")
        d = torch.empty((groups * a.shape[1], b.shape[1]), dtype=torch.bfloat16, device=a.device)
        problems.append((a.data_ptr(), a.stride(0), b.data_ptr(), b.stride(0), d.data_ptr(), d.stride(0), a.shape[1], b.shape[1]))
        outs.append(d)
    maps = torch.empty(groups * 512, dtype=torch.uint8, device=a0.device)          # the kernel's descriptors
    C.gemm_grouped_wgrad(problems[0], problems[1], row_off.data_ptr(), groups, rows, maps.data_ptr(), status_words().data_ptr(),
                         stream_handle())
    count_launch(2)
    return outs[0], outs[1]


def _version(t: torch.Tensor) -> Optional[int]:
    return None if t.is_inference() else t._version        # tensors made in inference mode count no versions


class MoEExchange:
    """Buffers and kernels of one expert-parallel MoE layer shape.  ``recv_q`` and ``recv_s`` hold what the last ``dispatch`` brought."""

    def __init__(self, eng: Engine, tokens: int, hidden: int, n_experts: int, topk: int, capacity_factor: float = 2.0,
                 blocks: Optional[int] = None, flag_lane: int = 5):
        if n_experts % eng.world or hidden % 128 or topk > 8:
            raise ValueError("MoEExchange: experts must divide over ranks, hidden % 128 == 0, top-k <= 8")
        self.eng, self.T, self.H, self.E, self.K = eng, tokens, hidden, n_experts, topk
        self.epr = n_experts // eng.world
        self.cap = int(capacity_factor * tokens * topk) // 128 * 128 + 128
        self.recv_q = eng.symmetric_tensor((self.cap, hidden), torch.uint8)
        self.recv_s = eng.symmetric_tensor((self.cap, hidden // 128), torch.float32)
        self.y = eng.symmetric_tensor((self.cap, hidden), torch.bfloat16)
        self.counts_all = eng.symmetric_tensor((eng.world, n_experts), torch.int32)
        self.x_bf16 = torch.empty((self.cap, hidden), dtype=torch.bfloat16, device="cuda")
        # de-duplicated exchange: where a row's payload is (alias), the rows and gate weights of a token's group on this
        # rank (64 bytes per row), and the groups' weighted sums of expert outputs
        self.alias = eng.symmetric_tensor((self.cap,), torch.int32)
        self.groups = eng.symmetric_tensor((self.cap, 16), torch.int32)
        self.z = eng.symmetric_tensor((self.cap, hidden), torch.bfloat16)
        self.alias.copy_(torch.arange(self.cap, dtype=torch.int32, device="cuda"))
        self.epoch = 0
        self._delivered = None             # (weak reference, version) of the rows if ``deliver`` wrote them past the receive buffers
        self.blocks = blocks or min(C.sm_count(), C.MAX_BLOCKS_PER_COLL)
        self.flag_lane = flag_lane

    # ---- routing -----------------------------------------------------------------------------
    @staticmethod
    def route(gate_logits: torch.Tensor, topk: int) -> Tuple[torch.Tensor, torch.Tensor]:
        probs = torch.softmax(gate_logits.float(), dim=-1)
        p, ids = probs.topk(topk, dim=-1)
        return ids.to(torch.int32), p.contiguous()

    def plan(self, ids: torch.Tensor) -> Dict[str, torch.Tensor]:
        """Where every (token, k) assignment lands: its row in the destination rank's receive buffer."""
        eng, E, epr = self.eng, self.E, self.epr
        flat = ids.reshape(-1).long()
        counts = torch.bincount(flat, minlength=E).to(torch.int32)
        if eng.world > 1:
            coll.all_gather(eng, counts, self.counts_all.view(-1), lane=self.flag_lane)
            counts_all = self.counts_all
        else:
            counts_all = counts.view(1, E)
        ca = counts_all.long()
        per_expert = ca.sum(0)                                     # rows each expert receives
        grp = per_expert.view(eng.world, epr)
        expert_base = (grp.cumsum(1) - grp).reshape(-1)            # start of the expert's segment on its rank
        src_prefix = (ca.cumsum(0) - ca)[eng.rank]                 # rows of lower ranks inside that segment
        order = torch.argsort(flat, stable=True)
        starts = counts.long().cumsum(0) - counts.long()
        pos_sorted = torch.arange(flat.numel(), device=flat.device) - starts[flat[order]]
        pos = torch.empty_like(pos_sorted)
        pos[order] = pos_sorted
        rows = expert_base[flat] + src_prefix[flat] + pos
        rows = torch.where(rows < self.cap, rows, torch.full_like(rows, -1)).to(torch.int32).view_as(ids)
        mine = grp[eng.rank]
        row_off = torch.zeros(epr + 1, dtype=torch.int32, device=ids.device)
        row_off[1:] = mine.cumsum(0).clamp(max=self.cap).to(torch.int32)
        return {"rows": rows.contiguous(), "row_off": row_off, "n_rows": row_off[-1:].contiguous()}

    def route_and_plan(self, gate_logits: torch.Tensor):
        """Fused routing: one kernel does softmax + top-k + per-expert counting (an assignment's position inside
        its expert's segment is the value its atomic increment returned), the counts are all-gathered, and a
        second kernel turns counts into receive rows.  Returns (ids, probs, plan)."""
        eng, T, K, E = self.eng, self.T, self.K, self.E
        dev = gate_logits.device
        lg = gate_logits.float().contiguous()
        ids = torch.empty((T, K), dtype=torch.int32, device=dev)
        probs = torch.empty((T, K), dtype=torch.float32, device=dev)
        pos = torch.empty((T, K), dtype=torch.int32, device=dev)
        counts = torch.zeros(E, dtype=torch.int32, device=dev)
        s = stream_handle()
        C.moe_route(lg.data_ptr(), ids.data_ptr(), probs.data_ptr(), pos.data_ptr(), counts.data_ptr(), T, E, K, s)
        if eng.world > 1:
            coll.all_gather(eng, counts, self.counts_all.view(-1), lane=self.flag_lane)
            counts_all = self.counts_all
        else:
            counts_all = counts
        rows = torch.empty((T, K), dtype=torch.int32, device=dev)
        row_off = torch.empty(self.epr + 1, dtype=torch.int32, device=dev)
        C.moe_plan(counts_all.data_ptr(), ids.data_ptr(), pos.data_ptr(), rows.data_ptr(), row_off.data_ptr(), eng.world, eng.rank, E,
                   T, K, self.cap, s)
        count_launch(2)
        return ids, probs, {"rows": rows, "row_off": row_off, "n_rows": row_off[-1:]}

    def route_backward(self, gate_logits: torch.Tensor, ids: torch.Tensor, dprobs: torch.Tensor) -> torch.Tensor:
        """Gradient (fp32) of the gate logits from the gradients ``dprobs`` (fp32 [tokens, topk]) of the probabilities of the experts
        ``ids``: the chain rule through the softmax over all experts."""
        lg = gate_logits.float().contiguous()
        out = torch.empty_like(lg)
        C.moe_route_backward(lg.data_ptr(), ids.data_ptr(), dprobs.data_ptr(), out.data_ptr(), lg.shape[0], self.E, self.K, stream_handle())
        count_launch()
        return out

    # ---- kernels ----------------------------------------------------------------------------
    def _exchange(self, kind: str, x, ids, rows, probs, out, gate=None, dedupe: bool = False) -> None:
        self.epoch += 1
        if kind == "dispatch":
            self._delivered = None
        st = status_words()
        off = self.eng.heap_offset
        C.moe_exchange(kind, self.eng.raw, [], 0, self.T, self.H, self.K, self.epr, off(self.recv_q),
                       off(self.recv_s), off(self.y), self.epoch, self.flag_lane,
                       [x.data_ptr()] if x is not None else [], [ids.data_ptr()], [rows.data_ptr()],
                       [probs.data_ptr()] if probs is not None else [], [out.data_ptr()] if out is not None else [],
                       [st.data_ptr()], self.blocks, 0, stream_handle(),
                       alias_off=off(self.alias), group_off=off(self.groups), z_off=off(self.z),
                       gate=[gate.data_ptr()] if gate is not None else [], dedupe=dedupe)
        count_launch()

    def dispatch(self, x: torch.Tensor, ids: torch.Tensor, plan: Dict[str, torch.Tensor], probs: Optional[torch.Tensor] = None,
                 gate: Optional[torch.Tensor] = None) -> None:
        """Rows of ``x`` go to the ranks of their experts (e4m3 + block scales).  With ``probs`` destination k of token t
        receives ``probs[t, k] * x[t]`` (how the backward pass sends gate-weighted output gradients).

        With ``gate`` (the routing probabilities; not together with ``probs``) a token crosses NVLink once per destination
        RANK instead of once per expert: the first of its assignments to a rank carries the row, the others are told
        where it is (``received`` / ``experts`` copy it locally while they convert to bf16), and the rank gets the list of
        the token's rows with their gate weights, which ``combine(..., grouped=True)`` needs."""
        if gate is not None and probs is not None:
            raise ValueError("MoEExchange.dispatch: gate (de-duplicated rows) and probs (scaled rows) exclude one another")
        if gate is not None and (gate.dtype != torch.float32 or gate.shape != ids.shape or not gate.is_contiguous()):
            raise ValueError("MoEExchange.dispatch: gate must be a contiguous fp32 [tokens, topk] tensor")
        self._exchange("dispatch", x, ids, plan["rows"], probs, None, gate=gate, dedupe=gate is not None)

    def received(self, plan: Dict[str, torch.Tensor], out: Optional[torch.Tensor] = None) -> torch.Tensor:
        """The rows that were last delivered to this rank, by ``dispatch`` or inside ``forward`` or a layer's pass, as bf16 [cap, hidden]
        (rows past the plan's count are not written)."""
        if self._delivered is not None:
            return self._received_past_buffers(plan, out)
        if out is None:
            out = torch.empty((self.cap, self.H), dtype=torch.bfloat16, device="cuda")
        C.moe_dequant(self.recv_q.data_ptr(), self.recv_s.data_ptr(), out.data_ptr(), plan["n_rows"].data_ptr(), self.cap,
                      self.H, stream_handle(), alias=self.alias.data_ptr())
        count_launch()
        return out

    def _received_past_buffers(self, plan: Dict[str, torch.Tensor], out: Optional[torch.Tensor]) -> torch.Tensor:
        """``received`` where ``deliver`` wrote the rows at once: ``recv_q`` and ``recv_s`` hold those of an earlier dispatch."""
        ref, version = self._delivered
        rows = ref()
        if rows is None or version != _version(rows):
            raise RuntimeError("MoEExchange.received: the rows that were last delivered are gone (their tensor was released or written to); "
                               "dispatch them again")
        if out is None:
            return rows.clone()
        if out.data_ptr() != rows.data_ptr():
            taken = torch.arange(self.cap, device=rows.device)[:, None] < plan["n_rows"]
            out.copy_(torch.where(taken, rows, out))
        return out

    def deliver(self, x: torch.Tensor, ids: torch.Tensor, plan: Dict[str, torch.Tensor], probs: Optional[torch.Tensor] = None,
                out: Optional[torch.Tensor] = None) -> torch.Tensor:
        """``dispatch`` and ``received`` in one.  In a world of one nothing travels and one kernel writes the rows; ``recv_q`` and
        ``recv_s`` stay as they are, and ``received`` finds the rows in the tensor returned here as long as that lives unchanged."""
        if self.eng.world > 1:
            self.dispatch(x, ids, plan, probs=probs)
            return self.received(plan, out)
        if out is None:
            out = torch.empty((self.cap, self.H), dtype=torch.bfloat16, device="cuda")
        C.moe_expand(x.data_ptr(), ids.data_ptr(), plan["rows"].data_ptr(), 0 if probs is None else probs.data_ptr(), out.data_ptr(), self.T, self.K,
                     self.H, stream_handle())
        count_launch()
        self._delivered = weakref.ref(out), _version(out)
        return out

    def combine_dot(self, g: torch.Tensor, ids: torch.Tensor, plan: Dict[str, torch.Tensor]) -> torch.Tensor:
        """``dot[t, k] = <g[t], y row of assignment (t, k)>`` (fp32 [tokens, topk]): with ``g`` the upstream gradient and
        the expert outputs of the forward pass still in ``self.y``, the gradient of the gate weights."""
        # a barrier between ranks that gives up leaves the rows unwritten: zeros then; a world of one has none and writes every value
        make = torch.zeros if self.eng.world > 1 else torch.empty
        out = make((self.T, self.K), dtype=torch.float32, device=g.device)
        self._exchange("combine_dot", g, ids, plan["rows"], None, out)
        return out

    def experts(self, w1: torch.Tensor, w2: torch.Tensor, plan: Dict[str, torch.Tensor]) -> None:
        """w1: [experts_per_rank * d_ff, hidden], w2: [experts_per_rank * hidden, d_ff]; result in self.y."""
        self.received(plan, self.x_bf16)
        self._experts(w1, w2, plan)

    def _experts(self, w1: torch.Tensor, w2: torch.Tensor, plan: Dict[str, torch.Tensor]) -> None:
        d_ff = w1.shape[0] // self.epr
        h = grouped_gemm(self.x_bf16, w1, plan["row_off"], d_ff, gelu=True)
        grouped_gemm(h, w2, plan["row_off"], self.H, out=self.y)

    def combine(self, ids: torch.Tensor, probs: Optional[torch.Tensor], plan: Dict[str, torch.Tensor], out: Optional[torch.Tensor] = None,
                grouped: bool = False) -> torch.Tensor:
        """``out[t] = sum_k probs[t, k] * (expert output of assignment (t, k))``, the rows pulled over NVLink; without ``probs`` the plain sum.

        ``grouped`` (after a dispatch with ``gate=probs``): every rank first adds up, locally, the weighted outputs of
        the assignments that one token has on it, and the token then pulls one row per rank instead of one per expert."""
        if out is None:
            out = torch.empty((self.T, self.H), dtype=torch.bfloat16, device="cuda")
        if grouped:
            C.moe_reduce_groups(self.y.data_ptr(), self.z.data_ptr(), self.alias.data_ptr(), self.groups.data_ptr(),
                                plan["n_rows"].data_ptr(), self.cap, self.H, stream_handle())
            count_launch()
        self._exchange("combine", None, ids, plan["rows"], probs, out, dedupe=grouped)
        return out

    def forward(self, x: torch.Tensor, gate_logits: torch.Tensor, w1: torch.Tensor, w2: torch.Tensor) -> torch.Tensor:
        ids, probs, plan = self.route_and_plan(gate_logits)
        # Adding up a token's rows on each rank before they travel saves NVLink traffic.  In a world of one nothing travels and it
        # would be a second pass over the sums: the combine weighs the expert rows itself (the same fp32 sum in the same order).
        grouped = self.eng.world > 1
        if grouped:
            self._exchange("dispatch", x, ids, plan["rows"], None, None, gate=probs, dedupe=True)
            self.experts(w1, w2, plan)
        else:
            self.deliver(x, ids, plan, out=self.x_bf16)
            self._experts(w1, w2, plan)
        return self.combine(ids, probs, plan, grouped=grouped)
