"""Attention backward dispatch.

Given ``dout`` and what the forward saved (q, k, v, o and the per-row logsumexp) this
produces dq, dk, dv.  On CUDA the tcgen05 backward kernel is used when the library
exports it; otherwise the gradients come from a library attention kernel
(``torch`` scaled-dot-product attention re-run under autograd), which is the A/B
baseline and the interim path.  On CPU a plain fp32 recomputation is used.
"""
from __future__ import annotations

import torch
import torch.nn.functional as F

import ctypes as C

from . import native
from .native import call, ptr, stream

native.register_signature("mb_attn_bwd_set_variant", [C.c_int], None)
native.register_signature("mb_attn_bwd_last_variant", [], C.c_int)


def _reference(dout, q, k, v, scale, causal, seqlens=(None, None)):
    from .functional import _ref_attention
    qq, kk, vv = (t.detach().float().requires_grad_(True) for t in (q, k, v))
    with torch.enable_grad():
        out, _ = _ref_attention(qq, kk, vv, scale, causal, *seqlens)
    dq, dk, dv = torch.autograd.grad(out, (qq, kk, vv), dout.float())
    return dq.to(q.dtype), dk.to(k.dtype), dv.to(v.dtype)


def _library(dout, q, k, v, scale, causal):
    qq, kk, vv = (t.detach().requires_grad_(True) for t in (q, k, v))
    with torch.enable_grad():
        out = F.scaled_dot_product_attention(
            qq.transpose(1, 2), kk.transpose(1, 2), vv.transpose(1, 2), is_causal=causal, scale=scale,
            enable_gqa=(q.shape[2] != k.shape[2]))
    return torch.autograd.grad(out, (qq, kk, vv), dout.transpose(1, 2))


def has_native_backward() -> bool:
    lib = native.kernels()
    return lib is not None and hasattr(lib, "mb_attn_bwd")


def backward(dout, q, k, v, o, lse, scale, causal, out=None, seqlens=(None, None)):
    """Returns (dq, dk, dv); with ``out=(dq, dk, dv)`` writes into those (possibly strided) views.
    ``seqlens``: (per-sample query lengths, per-sample key lengths) of a right-padded batch, or Nones."""
    padded = seqlens[0] is not None or seqlens[1] is not None
    if not q.is_cuda or (padded and not has_native_backward()):
        grads = _reference(dout, q, k, v, scale, causal, seqlens)
    elif has_native_backward():
        from .functional import Settings
        if Settings.attn_backend == "tcgen05":
            g = q.shape[2] // k.shape[2]
            if g == 1:
                return _native_backward(dout, q, k, v, o, lse, scale, causal, out, seqlens)
            if not Settings.attn_bwd_pipelined:    # that kernel knows no groups: every query head gets its own copy
                k, v = k.repeat_interleave(g, dim=2), v.repeat_interleave(g, dim=2)
            unit = _unit_heads(q, k) if Settings.attn_bwd_pipelined else 1
            if unit == g:
                return _native_backward(dout, q, k, v, o, lse, scale, causal, out, seqlens, unit)
            b, sk, nkv, d = k.shape if Settings.attn_bwd_pipelined else (*k.shape[:2], k.shape[2] // g, k.shape[3])
            if out is None:
                out = (torch.empty_like(q, memory_format=torch.contiguous_format),
                       *(torch.empty(b, sk, nkv, d, dtype=q.dtype, device=q.device) for _ in range(2)))
            dq, dk, dv = out
            part_k, part_v = (torch.empty(b, sk, nkv * (g // unit), d, dtype=q.dtype, device=q.device) for _ in range(2))
            _native_backward(dout, q, k, v, o, lse, scale, causal, (dq, part_k, part_v), seqlens, unit)
            call("mb_attn_sum_parts", ptr(part_k), ptr(part_v), ptr(dk), ptr(dv), b, sk, nkv, g // unit, d,
                 dk.stride(0), dk.stride(1), dk.stride(2), dv.stride(0), dv.stride(1), dv.stride(2), stream())
            return out
        else:
            grads = _reference(dout, q, k, v, scale, causal, seqlens) if padded else _library(dout, q, k, v, scale, causal)
    else:
        grads = _library(dout, q, k, v, scale, causal)
    if out is not None:
        for dst, src in zip(out, grads):
            dst.copy_(src)
        return out
    return grads


def _unit_heads(q, k) -> int:
    """Query heads of a group that one CTA sums into dK and dV.  A CTA's longest work item is that many walks over
    the queries; it must not exceed a CTA's share of the whole (148 CTAs, half of the blocks visible), or the last
    CTA works alone.  What is not summed inside a CTA costs a pass over dK and dV afterwards."""
    b, sq, nh, _ = q.shape
    g = nh // k.shape[2]
    most = (k.shape[1] + 127) // 128 * nh * b // 296
    return max((u for u in range(1, g + 1) if g % u == 0 and u <= most), default=1)


def _native_backward(dout, q, k, v, o, lse, scale, causal, out, seqlens=(None, None), unit_heads=1):
    b, sq, nh, d = q.shape
    sk = k.shape[1]
    if out is None:
        dq = torch.empty(b, sq, nh, d, dtype=q.dtype, device=q.device)
        dk = torch.empty(b, sk, nh // unit_heads, d, dtype=q.dtype, device=q.device)
        dv = torch.empty(b, sk, nh // unit_heads, d, dtype=q.dtype, device=q.device)
    else:
        dq, dk, dv = out
    dout = dout.contiguous()
    from .functional import Settings, _select_variant
    _select_variant("mb_attn_bwd_set_variant", 1 if Settings.attn_bwd_pipelined else 0)
    delta = torch.empty(b, nh, sq, dtype=torch.float32, device=q.device)
    dq_acc = torch.empty(b, nh, sq, d, dtype=torch.float32, device=q.device)   # zeroed by the launch wrapper
    call("mb_attn_bwd", ptr(dout), ptr(q), ptr(k), ptr(v), ptr(o), ptr(lse), ptr(delta), ptr(dq_acc),
         ptr(dq), ptr(dk), ptr(dv), b, sq, sk, nh, k.shape[2], unit_heads, d,
         q.stride(0), q.stride(1), q.stride(2), k.stride(0), k.stride(1), k.stride(2),
         v.stride(0), v.stride(1), v.stride(2),
         dq.stride(0), dq.stride(1), dq.stride(2), dk.stride(0), dk.stride(1), dk.stride(2),
         dv.stride(0), dv.stride(1), dv.stride(2), float(scale), int(causal), ptr(seqlens[0]), ptr(seqlens[1]),
         stream())
    return dq, dk, dv
