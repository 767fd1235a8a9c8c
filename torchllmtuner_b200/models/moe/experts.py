"""Grouped experts and token dispatch on one rank (reference: llmtuner/models/common/moe/experts.py:73-343,
llmtuner/parallel/expert_parallel/token_dispatch.py:127-275).

Weights are kept in the native packed layout `w1_EFD` (gate), `w3_EFD` (up), `w2_EDF` (down). Token copies are
sorted by expert into 128-row aligned segments (padding rows are zero), which lets the grouped tcgen05 GEMM tile
without ever crossing an expert boundary in M (forward, dgrad) or in K (wgrad).
"""
from __future__ import annotations

import torch
import torch.nn as nn

from ... import ops
from ...ops import reference as ref
from ...ops.cuda_ext import load as _ext

SEG_ALIGN = 128
PLAN_MAX_EXPERTS = 512      # of the planning kernels


def padded_capacity(num_copies: int, num_experts: int) -> int:
    """Static upper bound of padded rows: every expert wastes at most SEG_ALIGN-1 rows."""
    cap = num_copies + num_experts * (SEG_ALIGN - 1)
    return -(-cap // SEG_ALIGN) * SEG_ALIGN


def plan_segments(flat_expert: torch.Tensor, num_experts: int):
    """From the expert id of each token copy: (dest_row [n] int64 in the padded layout, seg_offsets [E+1] int32,
    counts [E] int64). Copies of one expert keep their order. On the device three kernels and no host synchronisation."""
    if (flat_expert.is_cuda and flat_expert.dtype == torch.int64 and 1 <= num_experts <= PLAN_MAX_EXPERTS
            and not torch.jit.is_tracing()):             # a trace would record the kernels' results as constants
        return tuple(_ext().moe_plan(flat_expert.contiguous(), num_experts, SEG_ALIGN))
    counts = torch.bincount(flat_expert, minlength=num_experts)
    padded = (counts + (SEG_ALIGN - 1)) // SEG_ALIGN * SEG_ALIGN
    zero = counts.new_zeros(1)
    seg = torch.cat([zero, padded.cumsum(0)])
    start = torch.cat([zero, counts.cumsum(0)])[:-1]
    order = torch.argsort(flat_expert, stable=True)
    rank = torch.empty_like(order)
    rank[order] = torch.arange(order.numel(), device=order.device)
    dest = rank - start[flat_expert] + seg[:-1][flat_expert]
    return dest, seg.to(torch.int32), counts


def _rows_view(t: torch.Tensor) -> torch.Tensor:
    """`t` itself when the grouped kernels can read it (unit inner stride, rows and base on 16-byte boundaries), else a copy.
    The gradients of gate and up are the two halves of one buffer: copying them cost as much as a grouped product."""
    if t.dim() == 2 and t.stride(1) == 1 and t.stride(0) % 8 == 0 and t.stride(0) >= t.shape[1] and t.data_ptr() % 16 == 0:
        return t
    return t.clone(memory_format=torch.contiguous_format)


class _GroupedLinear(torch.autograd.Function):
    """y_i[seg g] = x[seg g] @ w_i[g]^T over 128-aligned row segments, for one or more weights that read the same rows (gate and
    up). The input gradient of the second weight is added by the product's epilogue (in fp32, one rounding) instead of by a
    pass over two finished gradients."""

    @staticmethod
    def forward(ctx, x, seg, *ws):
        ys = []
        for w in ws:
            ys.append(torch.empty(x.shape[0], w.shape[1], dtype=x.dtype, device=x.device))
            _ext().grouped_gemm(x, w, ys[-1], seg, False)
        ctx.save_for_backward(x, seg, *ws)
        return tuple(ys) if len(ys) > 1 else ys[0]

    @staticmethod
    def backward(ctx, *dys):
        x, seg, *ws = ctx.saved_tensors
        dx, dws = None, []
        for i, (dy, w) in enumerate(zip(dys, ws)):
            dy = _rows_view(dy)
            if ctx.needs_input_grad[0]:
                if dx is None:
                    dx = torch.empty(x.shape, dtype=x.dtype, device=x.device)
                    _ext().grouped_gemm(dy, w, dx, seg, True)
                else:
                    _ext().grouped_gemm(dy, w, dx, seg, True, True)
            if ctx.needs_input_grad[2 + i]:
                dws.append(torch.empty_like(w))
                _ext().grouped_wgrad(dy, x, dws[-1], seg, False)
            else:
                dws.append(None)
        return (dx, None, *dws)


def grouped_linears(x, seg_offsets, *ws):
    """Several grouped projections of the same rows; one autograd node on the device."""
    if x.is_cuda and x.dtype == torch.bfloat16:
        return _GroupedLinear.apply(x, seg_offsets, *ws)
    return tuple(grouped_linear(x, w, seg_offsets) for w in ws)


def grouped_linear(x, w, seg_offsets, counts=None):
    if x.is_cuda and x.dtype == torch.bfloat16:
        return _GroupedLinear.apply(x, seg_offsets, w)
    # CPU statement over the padded layout
    outs = x.new_zeros(x.shape[0], w.shape[1])
    seg = seg_offsets.tolist()
    for e in range(w.shape[0]):
        s, t = seg[e], seg[e + 1]
        if t > s:
            outs[s:t] = torch.nn.functional.linear(x[s:t], w[e])
    return outs


class _PermuteRows(torch.autograd.Function):
    """rows[dest[c]] = x[c // k], padding rows of every segment zero; backward sums the k copies of every token. Rows past the
    last segment of the statically sized buffer stay unwritten: every consumer stops at that segment's end."""

    @staticmethod
    def forward(ctx, x, dest, cap, k, seg, counts):
        rows = (torch.empty if dest.numel() else torch.zeros)(cap, x.shape[1], dtype=x.dtype, device=x.device)
        _ext().permute_rows(x.contiguous(), dest, rows, k, seg, counts)
        ctx.save_for_backward(dest)
        ctx.k, ctx.T = k, x.shape[0]
        return rows

    @staticmethod
    def backward(ctx, g):
        (dest,) = ctx.saved_tensors
        return _ext().combine_rows(g.contiguous(), dest, None, ctx.T, ctx.k), None, None, None, None, None


class _CombineRows(torch.autograd.Function):
    """out[t] = sum_j w[t, j] * y[dest[t * k + j]] in fp32."""

    @staticmethod
    def forward(ctx, y, weights, dest, T, k, seg, counts):
        w = weights.float().contiguous()
        ctx.save_for_backward(y, w, dest, seg, counts)
        ctx.k = k
        return _ext().combine_rows(y.contiguous(), dest, w, T, k)

    @staticmethod
    def backward(ctx, g):
        y, w, dest, seg, counts = ctx.saved_tensors
        dy, dw = _ext().combine_bwd(g, y.contiguous(), dest, w.reshape(-1), ctx.k, seg, counts)
        return dy, dw.view_as(w), None, None, None, None, None


class GroupedExperts(nn.Module):
    def __init__(self, num_experts: int, hidden: int, inter: int, dtype=None, device=None, implementation: str = "native",
                 swiglu_limit: float | None = None, glu_fn=None):
        super().__init__()
        # `glu_fn(gate, up) -> hidden` replaces silu(gate) * up (Kimi's bounded SituGLU); None keeps the fused kernel
        self.glu_fn = glu_fn
        self.num_experts, self.hidden, self.inter, self.implementation = num_experts, hidden, inter, implementation
        # asymmetric clamp before the gated activation: gate <= limit, |up| <= limit
        # (reference: llmtuner/models/deepseek/deepseek_v4/modeling.py:164-169)
        self.swiglu_limit = swiglu_limit
        self.w1_EFD = nn.Parameter(torch.empty(num_experts, inter, hidden, dtype=dtype, device=device))
        self.w3_EFD = nn.Parameter(torch.empty(num_experts, inter, hidden, dtype=dtype, device=device))
        self.w2_EDF = nn.Parameter(torch.empty(num_experts, hidden, inter, dtype=dtype, device=device))
        for p in (self.w1_EFD, self.w3_EFD, self.w2_EDF):
            p.is_expert = True

    def _clamp(self, g, u):
        if self.swiglu_limit is None:
            return g, u
        return g.clamp(max=self.swiglu_limit), u.clamp(min=-self.swiglu_limit, max=self.swiglu_limit)

    def forward(self, rows: torch.Tensor, seg_offsets: torch.Tensor) -> torch.Tensor:
        """rows: padded expert-major rows [R, D]; returns [R, D]."""
        if rows.shape[0] == 0:
            return rows.new_zeros(0, self.hidden) + 0.0 * (self.w1_EFD.sum() + self.w3_EFD.sum() + self.w2_EDF.sum())
        if self.implementation == "eager":
            seg = seg_offsets.tolist()
            out = rows.new_zeros(rows.shape[0], self.hidden)
            for e in range(self.w1_EFD.shape[0]):
                s, t = seg[e], seg[e + 1]
                if t > s:
                    g_, u_ = self._clamp(ops.linear(rows[s:t], self.w1_EFD[e]), ops.linear(rows[s:t], self.w3_EFD[e]))
                    h = ops.swiglu(g_, u_) if self.glu_fn is None else self.glu_fn(g_, u_)
                    out[s:t] = ops.linear(h, self.w2_EDF[e])
            return out
        g, u = self._clamp(*grouped_linears(rows, seg_offsets, self.w1_EFD, self.w3_EFD))
        # rows past the last segment of a statically sized receive buffer hold nothing: the kernels skip them
        limit = seg_offsets[-1:] if rows.is_cuda and seg_offsets.dtype == torch.int32 else None
        h = ops.swiglu(g, u, limit) if self.glu_fn is None else self.glu_fn(g, u)
        return grouped_linear(h, self.w2_EDF, seg_offsets)


class LocalTokenDispatcher:
    """All experts live on this rank: stable sort of the copies by expert, zero-padded 128-aligned segments,
    score-weighted fp32 combine."""

    def __init__(self, num_experts: int):
        self.num_experts = num_experts

    def dispatch(self, x: torch.Tensor, indices: torch.Tensor):
        T, k = indices.shape
        flat = indices.reshape(-1)
        dest, seg, counts = plan_segments(flat, self.num_experts)
        cap = padded_capacity(T * k, self.num_experts)
        if x.is_cuda and x.dtype == torch.bfloat16 and x.shape[1] % 8 == 0:
            rows = _PermuteRows.apply(x, dest, cap, k, seg, counts)
        else:
            tok = torch.arange(T * k, device=x.device) // k
            rows = x.new_zeros(cap, x.shape[1]).index_copy(0, dest, x.index_select(0, tok))
        return rows, seg, {"dest": dest, "T": T, "k": k, "seg": seg, "counts": counts}

    def combine(self, y: torch.Tensor, weights: torch.Tensor, state) -> torch.Tensor:
        T, k = state["T"], state["k"]
        if y.is_cuda and y.dtype == torch.bfloat16 and y.shape[1] % 8 == 0:
            return _CombineRows.apply(y, weights, state["dest"], T, k, state["seg"], state["counts"])
        g = y.index_select(0, state["dest"]).view(T, k, -1)
        return (g.float() * weights.float().unsqueeze(-1)).sum(1).to(y.dtype)


class RoutedExperts(nn.Module):
    """dispatch -> grouped experts -> combine (reference: experts.py:288-343)."""

    def __init__(self, experts: GroupedExperts, dispatcher=None):
        super().__init__()
        self.experts = experts
        self.dispatcher = dispatcher or LocalTokenDispatcher(experts.num_experts)

    def forward(self, x, weights, indices):
        timer = getattr(self, "dispatch_timer", None)
        if timer is None:
            rows, seg, state = self.dispatcher.dispatch(x, indices)
            y = self.experts(rows, seg)
            return self.dispatcher.combine(y, weights, state)
        with timer.span("dispatch"):
            rows, seg, state = self.dispatcher.dispatch(x, indices)
        y = self.experts(rows, seg)
        with timer.span("combine"):
            return self.dispatcher.combine(y, weights, state)
