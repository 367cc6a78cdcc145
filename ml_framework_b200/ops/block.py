"""A whole transformer block of the GPT or Llama kind as one autograd node whose forward and backward are one native call
each (``csrc/ops/block.cu``): the launches of the operators of :mod:`.functional`, but for the bias gradients, two of which
share a launch, without their host work. A step of a small model is bound by that work.

It serves blocks that are exactly what the models build: bf16 on the GPU, plain layers, every parameter trained and used once,
no hooks on the layers inside. Whatever differs runs operator by operator. It is off unless the caller asks for it
(:func:`whole_blocks`), which the training engine does for forward and backward (blocks may be recomputed there) where nothing
works on single operators of a block, that is without data-parallel sharding or reduction.
"""
from __future__ import annotations

import ctypes as C
import threading
from contextlib import contextmanager
from typing import Optional

import torch
from torch.nn.modules.module import _has_any_global_hook

from .. import _lib
from . import gemm as _gemm
from . import native
from .functional import _done, _sink

_state = threading.local()
_BIASES = frozenset((1, 3, 5, 7, 9, 11))      # places of the parameters that a gated block lacks


@contextmanager
def whole_blocks(on: bool = True):
    """Blocks that are run inside (by this thread) may be one autograd node each."""
    before = getattr(_state, "on", False)
    _state.on = on
    try:
        yield
    finally:
        _state.on = before


class _Args(C.Structure):
    """MlfBlockArgs of csrc/mlf_api.h."""
    _fields_ = ([(n, C.c_int) for n in ("B", "S", "d", "Hq", "Hkv", "ff", "gated", "causal", "accumulate")] +
                [(n, C.c_float) for n in ("eps1", "eps2", "rope_theta", "scale")] +
                [(n, C.c_void_p) for n in (
                    "g1", "b1", "wqkv", "bqkv", "wo", "bo", "g2", "b2", "w1", "bb1", "w2", "bb2", "pos",
                    "x", "h1", "qkv", "a", "x1", "h2", "pre", "act", "mean1", "rstd1", "mean2", "rstd2", "lse", "y",
                    "dy", "wide", "row", "da", "dx1", "dx",
                    "dg1", "db1", "dwqkv", "dbqkv", "dwo", "dbo", "dg2", "db2", "dw1", "dbb1", "dw2", "dbb2",
                    "norm_scratch", "colsum_scratch", "flash_scratch")])


def _ptr(t: Optional[torch.Tensor]):
    return None if t is None else t.data_ptr()


def _takes_gradient(tgt: torch.Tensor, p: torch.Tensor) -> bool:
    return tgt.dtype is torch.bfloat16 and tgt.shape == p.shape and tgt.is_contiguous() and tgt.data_ptr() % 16 == 0 and tgt.device == p.device


class _BlockFn(torch.autograd.Function):
    @staticmethod
    def _saved(rows, stats, T, d, w, q, n1, gated):
        """Addresses of h1, qkv, a, x1, h2, pre, act and of mean1, rstd1, mean2, rstd2, lse."""
        at, out = rows.data_ptr(), []
        for cols in (d, w, q, d, d, n1):
            out.append(at)
            at += 2 * T * cols
        out.append(at)
        f = stats.data_ptr()
        return out + [None if gated else f, f + 4 * T, None if gated else f + 8 * T, f + 12 * T, f + 16 * T]

    @staticmethod
    def forward(ctx, x, positions, dims, *params):
        B, S, d, Hq, Hkv, ff, gated, causal, eps1, eps2, theta = dims
        T, q, w, n1 = B * S, Hq * 128, (Hq + 2 * Hkv) * 128, 2 * ff if gated else ff
        # h1 | qkv | a | x1 | h2 | pre | act, and the fp32 statistics: kept for the backward as the operators keep them
        rows = torch.empty(T * (3 * d + w + q + n1 + ff), dtype=torch.bfloat16, device=x.device)
        stats = torch.empty(4 * T + B * Hq * S, dtype=torch.float32, device=x.device)
        y = torch.empty_like(x)
        args = _Args(B, S, d, Hq, Hkv, ff, gated, causal, 0, eps1, eps2, theta, 128 ** -0.5, *[_ptr(p) for p in params], _ptr(positions),
                     x.data_ptr(), *_BlockFn._saved(rows, stats, T, d, w, q, n1, gated), y.data_ptr())
        rc = _lib.get().mlf_block_forward(C.byref(args), C.c_uint64(_lib.stream_handle()))
        if rc:
            _lib.check(rc, "mlf_block_forward")
        ctx.save_for_backward(x, positions, rows, stats, *params)
        ctx.dims, ctx.refs = dims, params
        return y

    @staticmethod
    def backward(ctx, dy):
        x, positions, rows, stats, *params = ctx.saved_tensors
        B, S, d, Hq, Hkv, ff, gated, causal, eps1, eps2, theta = ctx.dims
        T, q, w, n1 = B * S, Hq * 128, (Hq + 2 * Hkv) * 128, 2 * ff if gated else ff
        dev = x.device
        dy = dy.contiguous()
        if dy.data_ptr() % 16:
            dy = dy.clone()
        targets, temps, accumulate = [], {}, 0
        for i, p in enumerate(ctx.refs):
            if p is None:
                targets.append(None)
                continue
            tgt, acc = _sink(p)
            if tgt is None or not _takes_gradient(tgt, p):
                tgt, acc = torch.empty(p.shape, dtype=torch.bfloat16, device=dev), False
                temps[i] = tgt
            targets.append(tgt.data_ptr())
            accumulate |= int(acc) << i
        L = _lib.get()
        wide = max(n1, w)
        work = torch.empty(T * (wide + 2 * d + q), dtype=torch.bfloat16, device=dev)      # wide | row | dx1 | da
        dx = torch.empty_like(x)
        wp = work.data_ptr()
        row = wp + 2 * T * wide
        L.mlf_norm_bwd_scratch_elems.restype = L.mlf_flash_bwd_scratch_bytes.restype = C.c_longlong
        norm = native.scratch("norm_bwd", L.mlf_norm_bwd_scratch_elems(T, d) * 4, dev)
        flash = native.scratch("flash_bwd", L.mlf_flash_bwd_scratch_bytes(B, S, Hq), dev)
        col = None if gated else native.colsum_scratch(T, ((d, w), (d, n1)), dev)
        args = _Args(B, S, d, Hq, Hkv, ff, gated, causal, accumulate, eps1, eps2, theta, 128 ** -0.5, *[_ptr(p) for p in params], _ptr(positions),
                     x.data_ptr(), *_BlockFn._saved(rows, stats, T, d, w, q, n1, gated), None, dy.data_ptr(), wp, row,
                     row + 4 * T * d, row + 2 * T * d, dx.data_ptr(), *targets, norm.data_ptr(), _ptr(col), flash.data_ptr())
        rc = L.mlf_block_backward(C.byref(args), C.c_uint64(_lib.stream_handle()))
        if rc:
            _lib.check(rc, "mlf_block_backward")
        grads = []
        for i, p in enumerate(ctx.refs):
            g = temps.get(i)
            tgt, acc = _sink(p)
            if g is not None and tgt is not None:          # a buffer of another type or layout
                tgt.copy_(tgt + g if acc else g)
                g = None
            if p is not None and tgt is not None:
                _done(p)
            grads.append(g)
        return (dx if ctx.needs_input_grad[0] else None, None, None, *grads)


def _plain(m) -> bool:
    """Calling this layer runs its class's forward and nothing else."""
    return not (m._forward_hooks or m._forward_pre_hooks or m._backward_hooks or m._backward_pre_hooks or "forward" in m.__dict__)


def block(norm1, attn, norm2, mlp, first, second, x, positions, gated: bool):
    """The output of a pre-norm block, or None where it has to run operator by operator. ``first`` and ``second`` are the
    MLP's projections; the classes of the layers are the caller's to check."""
    if not getattr(_state, "on", False) or not torch.is_grad_enabled():
        return None
    if not (x.is_cuda and x.dtype is torch.bfloat16 and x.dim() == 3 and x.is_contiguous() and x.requires_grad and x.data_ptr() % 16 == 0):
        return None
    B, S, d = x.shape
    qkv, proj = attn.qkv, attn.proj
    if _has_any_global_hook() or not (_plain(attn) and _plain(qkv) and _plain(proj) and _plain(mlp)) or _gemm._piggyback is not None:
        return None
    Hq, Hkv = attn.n_heads, attn.n_kv_heads
    w, ff = (Hq + 2 * Hkv) * 128, second.weight.shape[1]
    if attn.head_dim != 128 or B * S == 0 or d % 256 or ff % 64 or (attn.rope_theta is None) == gated or x.device.index != torch._C._cuda_getDevice():
        return None
    params = (norm1.weight, None if gated else norm1.bias, qkv.weight, qkv.bias, proj.weight, proj.bias, norm2.weight,
              None if gated else norm2.bias, first.weight, first.bias, second.weight, second.bias)
    if len({id(p) for p in params if p is not None}) < (6 if gated else 12):
        return None                # one used twice: its second gradient has to find the first in the buffer
    n1 = 2 * ff if gated else ff
    shapes = ((d,), (d,), (w, d), (w,), (d, Hq * 128), (d,), (d,), (d,), (n1, d), (n1,), (d, ff), (d,))
    for i, (p, shape) in enumerate(zip(params, shapes)):
        if gated and i in _BIASES:
            if p is not None:
                return None
            continue
        if p is None or not (p.dtype is torch.bfloat16 and p.requires_grad and p.shape == shape and p.is_contiguous() and p.device == x.device
                             and p.data_ptr() % 16 == 0):
            return None
        mg = getattr(p, "main_grad", None)
        if mg is not None and not _takes_gradient(mg, p):
            return None
    if gated:
        if positions is None:
            positions = torch.arange(S, device=x.device).repeat(B)
        elif positions.dim() != 1 or positions.shape[0] != B * S or positions.dtype != torch.int64 or not positions.is_contiguous():
            return None
    dims = (B, S, d, Hq, Hkv, ff, int(gated), int(attn.causal), norm1.eps, norm2.eps, attn.rope_theta or 0.0)
    return _BlockFn.apply(x, positions if gated else None, dims, *params)
