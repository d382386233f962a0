"""Grouped (per-expert) linear layers on the tcgen05 GEMM kernel.

``grouped_linear(x, w[E, N, K], counts)``: rows of ``x`` are grouped by expert (``counts[e]`` rows
for expert ``e``); returns ``y`` with ``y_e = x_e @ w[e].T`` in the same row order.

The kernel works on a *padded* layout in which every expert's rows start at a multiple of 128
(the M tile) so that no output tile straddles two experts: rows are scattered into that layout
(padding rows are zero), the three GEMMs of forward / dgrad / wgrad run as single grouped
launches, and the result is gathered back.  Padding costs at most 127 rows per expert.
"""
from __future__ import annotations

import ctypes
from typing import List, Sequence, Tuple

import torch

from . import native

_BLOCK_M = 128
_bound = False


def _lib():
    global _bound
    lib = native.lib()
    if not _bound:
        vp, ci, c64 = ctypes.c_void_p, ctypes.c_int, ctypes.c_int64
        lib.hpb_gemm_bf16_grouped.argtypes = [vp, ci, c64, c64, vp, ci, c64, c64, vp, c64, ci, ci, ci, ci, ci, ci,
                                              vp, vp, ci, ci, vp, ci, vp]
        lib.hpb_gemm_bf16_grouped.restype = ci
        _bound = True
    return lib


def padded_layout(counts: Sequence[int], device) -> Tuple[torch.Tensor, torch.Tensor, torch.Tensor, int]:
    """``(row map [sum counts] -> padded row, block_group [blocks], group_offsets [E+1], padded rows)``."""
    offs = [0]
    blocks: List[int] = []
    rows: List[torch.Tensor] = []
    for e, c in enumerate(counts):
        pad = (c + _BLOCK_M - 1) // _BLOCK_M * _BLOCK_M
        rows.append(torch.arange(offs[-1], offs[-1] + c))
        blocks += [e] * (pad // _BLOCK_M)
        offs.append(offs[-1] + pad)
    row_map = torch.cat(rows).to(device) if rows else torch.zeros(0, dtype=torch.long, device=device)
    return (row_map, torch.tensor(blocks, dtype=torch.int32, device=device),
            torch.tensor(offs, dtype=torch.int32, device=device), offs[-1])


def _grouped(a, a_mn, a_rows, b, b_mn, b_rows, out, M, N, K, mode, block_group, group_offsets, E, b_group_rows,
             accumulate=False):
    dev = a.device
    rc = _lib().hpb_gemm_bf16_grouped(
        a.data_ptr(), a_mn, a.stride(0), a_rows, b.data_ptr(), b_mn, b.stride(0), b_rows,
        out.data_ptr(), out.stride(-2), int(out.dtype == torch.float32), int(accumulate), M, N, K, mode,
        native.ptr(block_group), native.ptr(group_offsets), E, b_group_rows,
        native.status_word(dev).data_ptr(), native.sm_count(dev), native.stream(dev))
    native.check(rc, "hpb_gemm_bf16_grouped")
    return out


class _GroupedLinear(torch.autograd.Function):
    @staticmethod
    def forward(ctx, x, w, counts):
        E, N, K = w.shape
        row_map, block_group, offsets, Mp = padded_layout(counts, x.device)
        xp = torch.zeros((Mp, K), dtype=x.dtype, device=x.device)
        xp.index_copy_(0, row_map, x)
        yp = torch.empty((Mp, N), dtype=x.dtype, device=x.device)
        if Mp > 0:
            _grouped(xp, False, Mp, w.view(E * N, K), False, E * N, yp, Mp, N, K, 1, block_group, None, E, N)
        ctx.save_for_backward(xp, w, row_map, block_group, offsets)
        ctx.dims = (E, N, K, Mp)
        return yp.index_select(0, row_map)

    @staticmethod
    def backward(ctx, dy):
        xp, w, row_map, block_group, offsets = ctx.saved_tensors
        E, N, K, Mp = ctx.dims
        dyp = torch.zeros((Mp, N), dtype=dy.dtype, device=dy.device)
        dyp.index_copy_(0, row_map, dy.contiguous())
        dx = dw = None
        if ctx.needs_input_grad[0]:
            dxp = torch.empty((Mp, K), dtype=dy.dtype, device=dy.device)
            if Mp > 0:
                # dx = dy @ W_e : B = W stacked [E*N, K], MN-major with the contraction along its rows
                _grouped(dyp, False, Mp, w.view(E * N, K), True, E * N, dxp, Mp, K, N, 1, block_group, None, E, N)
            dx = dxp.index_select(0, row_map)
        if ctx.needs_input_grad[1]:
            dw = torch.empty_like(w)
            # dW_e[N, K] = dy_e^T x_e : contraction over the expert's (padded, zero-filled) rows
            _grouped(dyp, True, Mp, xp, True, Mp, dw.view(E * N, K), N, K, 0, 2, None, offsets, E, 0)
        return dx, dw, None


def grouped_linear(x: torch.Tensor, w: torch.Tensor, counts: Sequence[int]) -> torch.Tensor:
    """``y_e = x_e @ w[e].T`` for rows grouped by expert; bf16 CUDA tensors."""
    assert x.dim() == 2 and w.dim() == 3 and x.shape[1] == w.shape[2]
    assert sum(counts) == x.shape[0] and len(counts) == w.shape[0]
    return _GroupedLinear.apply(x.contiguous(), w.contiguous(), list(int(c) for c in counts))


# ------------------------------------------------------------ local experts --
# Rows per expert (mean) from which the row-grouped products run on CTA pairs with 256-row padding; below
# it, on the 128 x 256 kernel with 128-row padding.  The pair tile runs at 1.18 times the rate but wastes
# 128 instead of 64 padding rows per expert on average: equal cost at (R + 128) / 1.18 = R + 64, R = 290.
# Measured, 16 experts of 7168 x 2048, forward + backward, pad 128 / 256: 64 rows 1.10 / 1.18 ms, 256 rows
# 1.60 / 1.64, 384 rows 2.09 / 2.06, 512 rows 2.63 / 2.47, 2048 rows 8.85 / 8.19.
_PAIR_MIN_ROWS = 290


def _local_lib():
    lib = native.lib()
    if not getattr(lib, "_hpb_moe_local_bound", False):
        vp, ci, c64 = ctypes.c_void_p, ctypes.c_int, ctypes.c_int64
        lib.hpb_gemm2_bf16_grouped.argtypes = [vp, c64, c64, vp, ci, c64, c64, vp, c64, ci, ci, ci, ci, vp, vp, vp, ci,
                                               ci, vp, ci, vp]
        lib.hpb_moe_count.argtypes = [vp, vp, vp, vp, vp, c64, ci, ci, vp]
        lib.hpb_moe_place.argtypes = [vp, vp, vp, vp, vp, vp, vp, c64, ci, ci, c64, vp, vp]
        lib.hpb_moe_gather.argtypes = [vp, vp, vp, c64, ci, ci, c64, vp, vp]
        lib.hpb_moe_combine.argtypes = [vp, vp, vp, vp, c64, ci, ci, c64, vp, vp]
        lib.hpb_moe_combine_bwd.argtypes = [vp, vp, vp, vp, vp, vp, c64, ci, ci, c64, vp, vp]
        lib._hpb_moe_local_bound = True
    return lib


def _expert_rows(a, w, out, block_group, pad, w_mn):
    """``out[rows of e] = a[rows of e] @ w[e].T`` (``w_mn``: ``@ w[e]``), rows padded to ``pad`` per expert."""
    E, rows_b = w.shape[0], w.shape[1]
    M, K = a.shape
    N = out.shape[1]
    dev = a.device
    if pad == _BLOCK_M:
        native.check(_lib().hpb_gemm_bf16_grouped(
            a.data_ptr(), 0, a.stride(0), M, w.data_ptr(), w_mn, w.stride(1), E * rows_b, out.data_ptr(), out.stride(0),
            0, 0, M, N, K, 1, block_group.data_ptr(), None, E, rows_b, native.status_word(dev).data_ptr(),
            native.sm_count(dev), native.stream(dev)), "hpb_gemm_bf16_grouped")
        return out
    native.check(_local_lib().hpb_gemm2_bf16_grouped(
        a.data_ptr(), a.stride(0), M, w.data_ptr(), w_mn, w.stride(1), E * rows_b, out.data_ptr(), out.stride(0),
        M, N, K, 1, block_group.data_ptr(), None, None, E, rows_b, native.status_word(dev).data_ptr(),
        native.sm_count(dev), native.stream(dev)), "hpb_gemm2_bf16_grouped")
    return out


def _expert_wgrad(a, b, out, table):
    """``out[e] = a[rows of e].T @ b[rows of e]``."""
    E, M, N = out.shape
    dev = a.device
    native.check(_local_lib().hpb_gemm2_bf16_grouped(
        a.data_ptr(), a.stride(0), a.shape[0], b.data_ptr(), 1, b.stride(0), b.shape[0], out.data_ptr(), N, M, N, 0, 2,
        None, table.data_ptr(), table.data_ptr() + 4 * E, E, 0, native.status_word(dev).data_ptr(), native.sm_count(dev),
        native.stream(dev)), "hpb_gemm2_bf16_grouped")
    return out


class _Plan:
    """Rows of a call: which padded row every (token, slot) pair takes.

    ``table``  [E] group starts, [E] group ends, [E] counts, 1 word: an id was out of range
    ``slots``  [rows / pad] expert of each row block, [rows] pair of each row (-1: padding), [pairs] row of
               each pair
    Both are handed to the kernels as addresses into them: a tensor view each would cost the host more
    than the launch."""

    def __init__(self, idx, num_experts):
        lib = _local_lib()
        dev = idx.device
        T, k = idx.shape
        E, pairs = num_experts, T * k
        pad = 256 if pairs >= _PAIR_MIN_ROWS * E else _BLOCK_M
        self.idx, self.dims = idx, (T, k, E, None, pad)
        self.hist = torch.empty((pairs + 255) // 256 * E, dtype=torch.int32, device=dev)
        self.table = torch.empty(3 * E + 1, dtype=torch.int32, device=dev)
        starts = self.table.data_ptr()
        native.check(lib.hpb_moe_count(idx.data_ptr(), self.hist.data_ptr(), starts + 8 * E, starts, starts + 4 * E,
                                       pairs, E, pad, native.stream(dev)), "hpb_moe_count")

    def place(self):
        """Read the per-expert counts back, which sizes the layout and refuses expert ids out of range, and
        fill ``slots``.  (The host work between the read-back and the first product is not hidden by anything.)"""
        T, k, E, _, pad = self.dims
        dev = self.idx.device
        *per_expert, bad = self.table[2 * E:].tolist()
        if bad:
            raise ValueError(f"expert ids must lie in [0, {E})")
        rows = sum((c + pad - 1) // pad * pad for c in per_expert)
        self.dims = (T, k, E, rows, pad)
        self.slots = torch.empty(rows // pad + rows + T * k, dtype=torch.int32, device=dev)
        starts = self.table.data_ptr()
        native.check(_local_lib().hpb_moe_place(
            self.idx.data_ptr(), self.hist.data_ptr(), starts, starts + 4 * E, self.slots.data_ptr(),
            _row_pair(self.slots, self.dims), _pos(self.slots, self.dims), T * k, E, pad, rows,
            native.status_word(dev).data_ptr(), native.stream(dev)), "hpb_moe_place")
        self.idx = self.hist = None


def _row_pair(slots, dims):
    return slots.data_ptr() + 4 * (dims[3] // dims[4])


def _pos(slots, dims):
    return _row_pair(slots, dims) + 4 * dims[3]


def _pos_tensor(slots, dims):
    """The row of every (token, slot) pair, for tensor operations."""
    T, k = dims[:2]
    return slots[slots.shape[0] - T * k:].view(T, k).long()


class _ExpertRows(torch.autograd.Function):
    """``yp[row of (t, j)] = expert_{idx[t, j]}(x[t])`` in the padded layout of the grouped GEMMs."""

    @staticmethod
    def forward(ctx, x, w_gate_up, w_down, plan):
        lib = _local_lib()
        dev = x.device
        stream = native.stream(dev)
        _, F2, H = w_gate_up.shape
        plan.place()
        T, k, E, rows, pad = plan.dims
        xp = torch.empty((rows, H), dtype=x.dtype, device=dev)
        native.check(lib.hpb_moe_gather(x.data_ptr(), _row_pair(plan.slots, plan.dims), xp.data_ptr(), rows, k, H,
                                        T * k, native.status_word(dev).data_ptr(), stream), "hpb_moe_gather")
        gu = torch.empty((rows, F2), dtype=x.dtype, device=dev)
        _expert_rows(xp, w_gate_up, gu, plan.slots, pad, False)
        act = torch.empty((rows, F2 // 2), dtype=x.dtype, device=dev)
        native.check(lib.hpb_swiglu_fwd(gu.data_ptr(), act.data_ptr(), rows, F2 // 2, native.sm_count(dev), stream),
                     "hpb_swiglu_fwd")
        yp = torch.empty((rows, H), dtype=x.dtype, device=dev)
        _expert_rows(act, w_down, yp, plan.slots, pad, False)
        ctx.save_for_backward(xp, gu, act, w_gate_up, w_down, plan.table, plan.slots)
        ctx.dims = plan.dims
        return yp

    @staticmethod
    def backward(ctx, dyp):
        xp, gu, act, w_gate_up, w_down, table, slots = ctx.saved_tensors
        T, k, E, rows, pad = ctx.dims
        lib = _local_lib()
        dev, dt = xp.device, xp.dtype
        stream = native.stream(dev)
        H, F2 = xp.shape[1], gu.shape[1]
        need_x, need_w1, need_w2 = ctx.needs_input_grad[:3]
        dyp = _rows16(dyp)
        dx = dw1 = dw2 = None
        if need_w2:
            dw2 = _expert_wgrad(dyp, act, torch.empty_like(w_down), table)
        if need_x or need_w1:
            dact = torch.empty_like(act)
            _expert_rows(dyp, w_down, dact, slots, pad, True)
            dgu = torch.empty_like(gu)
            native.check(lib.hpb_swiglu_bwd(gu.data_ptr(), dact.data_ptr(), dgu.data_ptr(), rows, F2 // 2,
                                            native.sm_count(dev), stream), "hpb_swiglu_bwd")
            if need_w1:
                dw1 = _expert_wgrad(dgu, xp, torch.empty_like(w_gate_up), table)
            if need_x:
                dxp = torch.empty((rows, H), dtype=dt, device=dev)
                _expert_rows(dgu, w_gate_up, dxp, slots, pad, True)
                dx = torch.empty((T, H), dtype=dt, device=dev)
                native.check(lib.hpb_moe_combine(dxp.data_ptr(), _pos(slots, ctx.dims), None, dx.data_ptr(), T, k, H,
                                                 rows, native.status_word(dev).data_ptr(), stream), "hpb_moe_combine")
        return dx, dw1, dw2, None


def _combine_rows(yp, gate, slots, dims):
    T, k, _, rows, _ = dims
    dev, H = yp.device, yp.shape[1]
    y = torch.empty((T, H), dtype=yp.dtype, device=dev)
    native.check(_local_lib().hpb_moe_combine(yp.data_ptr(), _pos(slots, dims), gate.data_ptr(), y.data_ptr(), T, k, H,
                                              rows, native.status_word(dev).data_ptr(), native.stream(dev)),
                 "hpb_moe_combine")
    return y


class _Combine(torch.autograd.Function):
    """``y[t] = sum_j gate[t, j] * yp[row of (t, j)]``.  A node of its own, so that the gate weights keep their
    higher derivatives (the products of the experts have none).  The backward pass multiplies with a private
    copy of the gate, which a caller may overwrite; ``gate`` itself stands for its history only."""

    @staticmethod
    def forward(ctx, yp, gate, plan):
        own = gate.to(torch.float32, copy=True, memory_format=torch.contiguous_format)
        ctx.save_for_backward(yp if ctx.needs_input_grad[1] else None, own, plan.slots)
        ctx.gate, ctx.version = gate, gate._version
        ctx.dims, ctx.like = plan.dims, (yp.dtype, yp.shape[1])
        return _combine_rows(yp, own, plan.slots, plan.dims)

    @staticmethod
    def backward(ctx, dy):
        yp, gate, slots = ctx.saved_tensors
        T, k, _, rows, _ = ctx.dims
        dtype, H = ctx.like
        need_rows, need_gate = ctx.needs_input_grad[:2]
        dyp = dgate = None
        if torch.is_grad_enabled() or not torch._C._has_storage(dy):
            # a graph of the gradients, or a batch of them, is wanted: the same sums as tensor operations
            if torch.is_grad_enabled():
                if ctx.gate._version != ctx.version:
                    raise RuntimeError("the gate weights were overwritten after the forward pass; a graph of their "
                                       "gradients needs them")
                gate = ctx.gate.float()
            pos = _pos_tensor(slots, ctx.dims)
            if need_rows:
                dyp = torch.zeros((rows, H), dtype=dtype, device=dy.device).index_copy(
                    0, pos.view(-1), (gate[:, :, None] * dy[:, None].float()).to(dtype).reshape(T * k, H))
            if need_gate:
                dgate = torch.stack([(dy.float() * yp.index_select(0, pos[:, j]).float()).sum(-1) for j in range(k)],
                                    -1).to(ctx.gate.dtype)
            return dyp, dgate, None
        dy = _rows16(dy)
        dyp = torch.empty((rows, H), dtype=dtype, device=dy.device)
        dgate = torch.empty((T, k), dtype=torch.float32, device=dy.device) if need_gate else None
        native.check(_local_lib().hpb_moe_combine_bwd(dy.data_ptr(), _row_pair(slots, ctx.dims), gate.data_ptr(),
                                                      native.ptr(yp), dyp.data_ptr(), native.ptr(dgate), rows, k, H,
                                                      T * k, native.status_word(dy.device).data_ptr(),
                                                      native.stream(dy.device)), "hpb_moe_combine_bwd")
        return dyp, dgate.to(ctx.gate.dtype) if need_gate else None, None


def _plain(t: torch.Tensor) -> bool:
    return type(t) in (torch.Tensor, torch.nn.Parameter)


def local_experts_usable(x, topk_idx, topk_w, w_gate_up, w_down, num_experts) -> bool:
    """Calls that ``local_experts`` serves; every other one takes the general formulation."""
    return (x.is_cuda and x.dtype == torch.bfloat16 and x.dim() == 2
            and all(map(_plain, (x, topk_idx, topk_w, w_gate_up, w_down)))
            and w_gate_up.dtype == w_down.dtype == torch.bfloat16 and w_gate_up.dim() == 3 and w_down.dim() == 3
            and w_gate_up.device == w_down.device == topk_idx.device == topk_w.device == x.device
            and topk_w.is_floating_point() and topk_w.shape == topk_idx.shape and topk_idx.dtype == torch.int64
            and topk_idx.shape[0] == x.shape[0] and 0 < topk_idx.numel() < 1 << 30 and w_gate_up.shape[0] == num_experts <= 8192
            and w_gate_up.shape[2] == x.shape[1] and w_gate_up.shape[1] % 16 == 0 and x.shape[1] % 8 == 0
            and w_down.shape == (num_experts, x.shape[1], w_gate_up.shape[1] // 2))


def local_experts(x, topk_idx, topk_w, w_gate_up, w_down):
    """``y[t] = sum_j topk_w[t, j] * expert_{topk_idx[t, j]}(x[t])`` with every expert on this GPU
    (``moe_local.cu`` around the grouped GEMMs)."""
    plan = _Plan(topk_idx.contiguous(), w_gate_up.shape[0])
    yp = _ExpertRows.apply(_rows16(x), _rows16(w_gate_up), _rows16(w_down), plan)
    if torch.autograd.forward_ad.unpack_dual(topk_w).tangent is not None:
        pos, gate = _pos_tensor(plan.slots, plan.dims), topk_w.float()
        return sum(gate[:, j, None] * yp.index_select(0, pos[:, j]).float() for j in range(pos.shape[1])).to(x.dtype)
    if torch.is_grad_enabled() and (yp.requires_grad or topk_w.requires_grad):
        return _Combine.apply(yp, topk_w, plan)
    return _combine_rows(yp, topk_w.to(torch.float32).contiguous(), plan.slots, plan.dims)


def _rows16(t: torch.Tensor) -> torch.Tensor:
    """``t`` contiguous on a 16-byte boundary (the kernels read whole 16-byte vectors)."""
    t = t.contiguous()
    return t if t.data_ptr() % 16 == 0 else t.clone()
