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
        a.data_ptr(), int(a_mn), a.stride(0), a_rows, b.data_ptr(), int(b_mn), b.stride(0), b_rows,
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
        lib.hpb_moe_place.argtypes = [vp, vp, vp, vp, vp, vp, vp, c64, ci, ci, vp]
        lib.hpb_moe_gather.argtypes = [vp, vp, vp, c64, ci, ci, vp]
        lib.hpb_moe_combine.argtypes = [vp, vp, vp, vp, c64, ci, ci, vp]
        lib.hpb_moe_combine_bwd.argtypes = [vp, vp, vp, vp, vp, vp, c64, ci, ci, vp]
        lib._hpb_moe_local_bound = True
    return lib


def _expert_rows(a, w, out, block_group, pad, w_mn):
    """``out[rows of e] = a[rows of e] @ w[e].T`` (``w_mn``: ``@ w[e]``), rows padded to ``pad`` per expert."""
    E, rows_b = w.shape[0], w.shape[1]
    M, K = a.shape
    N = out.shape[1]
    if pad == _BLOCK_M:
        return _grouped(a, False, M, w.view(E * rows_b, -1), w_mn, E * rows_b, out, M, N, K, 1, block_group, None, E,
                        rows_b)
    dev = a.device
    native.check(_local_lib().hpb_gemm2_bf16_grouped(
        a.data_ptr(), a.stride(0), M, w.data_ptr(), int(w_mn), w.stride(1), E * rows_b, out.data_ptr(), out.stride(0),
        M, N, K, 1, block_group.data_ptr(), None, None, E, rows_b, native.status_word(dev).data_ptr(),
        native.sm_count(dev), native.stream(dev)), "hpb_gemm2_bf16_grouped")
    return out


def _expert_wgrad(a, b, out, starts, ends):
    """``out[e] = a[rows of e].T @ b[rows of e]``."""
    E, M, N = out.shape
    dev = a.device
    native.check(_local_lib().hpb_gemm2_bf16_grouped(
        a.data_ptr(), a.stride(0), a.shape[0], b.data_ptr(), 1, b.stride(0), b.shape[0], out.data_ptr(), N, M, N, 0, 2,
        None, starts.data_ptr(), ends.data_ptr(), E, 0, native.status_word(dev).data_ptr(), native.sm_count(dev),
        native.stream(dev)), "hpb_gemm2_bf16_grouped")
    return out


class _LocalExperts(torch.autograd.Function):
    """``y[t] = sum_j gate[t, j] * expert_{idx[t, j]}(x[t])`` with every expert on this GPU
    (``moe_local.cu`` around the grouped GEMMs).  One read-back of the per-expert counts, which sizes
    the padded layout and refuses expert ids out of range."""

    @staticmethod
    def forward(ctx, x, gate, w_gate_up, w_down, idx):
        lib = _local_lib()
        dev = x.device
        stream = native.stream(dev)
        T, k = idx.shape
        E, F2, H = w_gate_up.shape
        pairs = T * k
        pad = 256 if pairs >= _PAIR_MIN_ROWS * E else _BLOCK_M
        gate_f = gate.detach().to(torch.float32).contiguous()
        hist = torch.empty((pairs + 255) // 256 * E, dtype=torch.int32, device=dev)
        table = torch.empty(3 * E + 1, dtype=torch.int32, device=dev)
        starts, ends, counts = table[:E], table[E:2 * E], table[2 * E:]
        native.check(lib.hpb_moe_count(idx.data_ptr(), hist.data_ptr(), counts.data_ptr(), starts.data_ptr(),
                                       ends.data_ptr(), pairs, E, pad, stream), "hpb_moe_count")
        *per_expert, bad = counts.tolist()
        if bad:
            raise ValueError(f"expert ids must lie in [0, {E})")
        rows = sum((c + pad - 1) // pad * pad for c in per_expert)
        slots = torch.empty(rows // pad + rows + pairs, dtype=torch.int32, device=dev)
        block_group, row_pair, pos = slots.split([rows // pad, rows, pairs])
        native.check(lib.hpb_moe_place(idx.data_ptr(), hist.data_ptr(), starts.data_ptr(), ends.data_ptr(),
                                       block_group.data_ptr(), row_pair.data_ptr(), pos.data_ptr(), pairs, E, pad,
                                       stream), "hpb_moe_place")
        xp = torch.empty((rows, H), dtype=x.dtype, device=dev)
        native.check(lib.hpb_moe_gather(x.data_ptr(), row_pair.data_ptr(), xp.data_ptr(), rows, k, H, stream),
                     "hpb_moe_gather")
        gu = torch.empty((rows, F2), dtype=x.dtype, device=dev)
        _expert_rows(xp, w_gate_up, gu, block_group, pad, False)
        act = torch.empty((rows, F2 // 2), dtype=x.dtype, device=dev)
        native.check(lib.hpb_swiglu_fwd(gu.data_ptr(), act.data_ptr(), rows, F2 // 2, native.sm_count(dev), stream),
                     "hpb_swiglu_fwd")
        yp = torch.empty((rows, H), dtype=x.dtype, device=dev)
        _expert_rows(act, w_down, yp, block_group, pad, False)
        y = torch.empty((T, H), dtype=x.dtype, device=dev)
        native.check(lib.hpb_moe_combine(yp.data_ptr(), pos.data_ptr(), gate_f.data_ptr(), y.data_ptr(), T, k, H,
                                         stream), "hpb_moe_combine")
        ctx.save_for_backward(xp, gu, act, yp if ctx.needs_input_grad[1] else None, gate_f, w_gate_up, w_down, table,
                              slots)
        ctx.dims = (T, k, E, rows, pad)
        ctx.gate_dtype = gate.dtype
        return y

    @staticmethod
    def backward(ctx, dy):
        xp, gu, act, yp, gate_f, w_gate_up, w_down, table, slots = ctx.saved_tensors
        T, k, E, rows, pad = ctx.dims
        lib = _local_lib()
        dev, dt = xp.device, xp.dtype
        stream = native.stream(dev)
        H, F2 = xp.shape[1], gu.shape[1]
        block_group, row_pair, pos = slots.split([rows // pad, rows, T * k])
        starts, ends = table[:E], table[E:2 * E]
        need_x, need_gate, need_w1, need_w2 = ctx.needs_input_grad[:4]
        dy = _rows16(dy)
        dyp = torch.empty((rows, H), dtype=dt, device=dev)
        dgate = torch.empty((T, k), dtype=torch.float32, device=dev) if need_gate else None
        native.check(lib.hpb_moe_combine_bwd(dy.data_ptr(), row_pair.data_ptr(), gate_f.data_ptr(), native.ptr(yp),
                                             dyp.data_ptr(), native.ptr(dgate), rows, k, H, stream),
                     "hpb_moe_combine_bwd")
        dx = dw1 = dw2 = None
        if need_w2:
            dw2 = _expert_wgrad(dyp, act, torch.empty_like(w_down), starts, ends)
        if need_x or need_w1:
            dact = torch.empty_like(act)
            _expert_rows(dyp, w_down, dact, block_group, pad, True)
            dgu = torch.empty_like(gu)
            native.check(lib.hpb_swiglu_bwd(gu.data_ptr(), dact.data_ptr(), dgu.data_ptr(), rows, F2 // 2,
                                            native.sm_count(dev), stream), "hpb_swiglu_bwd")
            if need_w1:
                dw1 = _expert_wgrad(dgu, xp, torch.empty_like(w_gate_up), starts, ends)
            if need_x:
                dxp = torch.empty((rows, H), dtype=dt, device=dev)
                _expert_rows(dgu, w_gate_up, dxp, block_group, pad, True)
                dx = torch.empty((T, H), dtype=dt, device=dev)
                native.check(lib.hpb_moe_combine(dxp.data_ptr(), pos.data_ptr(), None, dx.data_ptr(), T, k, H, stream),
                             "hpb_moe_combine")
        return dx, dgate.to(ctx.gate_dtype) if need_gate else None, dw1, dw2, None


def _plain(t: torch.Tensor) -> bool:
    return type(t) in (torch.Tensor, torch.nn.Parameter)


def local_experts_usable(x, topk_idx, topk_w, w_gate_up, w_down, num_experts) -> bool:
    """Calls that ``local_experts`` serves; every other one takes the general formulation."""
    return (x.is_cuda and x.dtype == torch.bfloat16 and x.dim() == 2 and all(map(_plain, (x, topk_w, w_gate_up, w_down)))
            and w_gate_up.dtype == w_down.dtype == torch.bfloat16 and w_gate_up.dim() == 3 and w_down.dim() == 3
            and w_gate_up.device == w_down.device == topk_idx.device == topk_w.device == x.device
            and topk_w.is_floating_point() and topk_w.shape == topk_idx.shape and topk_idx.dtype == torch.int64
            and topk_idx.shape[0] == x.shape[0] and topk_idx.numel() > 0 and w_gate_up.shape[0] == num_experts <= 8192
            and w_gate_up.shape[2] == x.shape[1] and w_gate_up.shape[1] % 16 == 0 and x.shape[1] % 8 == 0
            and w_down.shape == (num_experts, x.shape[1], w_gate_up.shape[1] // 2))


def local_experts(x, topk_idx, topk_w, w_gate_up, w_down):
    return _LocalExperts.apply(_rows16(x), topk_w, _rows16(w_gate_up), _rows16(w_down), topk_idx.contiguous())


def _rows16(t: torch.Tensor) -> torch.Tensor:
    """``t`` contiguous on a 16-byte boundary (the kernels read whole 16-byte vectors)."""
    t = t.contiguous()
    return t if t.data_ptr() % 16 == 0 else t.clone()
