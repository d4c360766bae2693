"""One decoding step through a stack of plain transformer blocks in one native call (csrc/decode_stack.cu).

:func:`stack_step` looks every block over (structure, types, hooks, dtypes) and hands the pointers of its weights and
caches to the library, which launches the whole stack.  Anything out of the ordinary -- parallel or cross-attention
blocks, tensor parallelism, hooks, a ``forward`` of an instance's own, dropout in training mode, other dtypes or shapes,
weights that are no parameters or live elsewhere, CPU tensors -- is answered with ``None`` and goes through the modules
one by one.
"""
from __future__ import annotations

import ctypes

import torch
from torch.nn.modules import module as nn_module

from ..models import transformer      # (imports this module in turn; its names are looked up when a step runs)
from ..modules import layers as L
from . import native
from .functional import Settings, rope_tables
from .native import ptr, stream

_PER_BLOCK = 13
_BF16 = torch.bfloat16
_Parameter = torch.nn.Parameter


def _tensors(mod, shape, device: int, out: list) -> bool:
    """Appends the addresses of ``mod``'s weight, of that shape, and of its bias (0: it has none); False where the
    kernels cannot read them.  (Looked at for every tensor of every step, so written out: a stack of 24 blocks is looked
    over in 215 us, in 300 with a loop over the names and imports in :func:`_block`.)"""
    ps = mod._parameters
    p = ps.get("weight")
    if (type(p) is not _Parameter or p.dtype is not _BF16 or p.shape != shape or not p.is_contiguous()
            or p.get_device() != device):
        return False                   # also where it is computed or replaced: not a parameter
    at = p.data_ptr()
    if at & 15 or not at:
        return False
    out.append(at)
    p = ps.get("bias")
    if p is None:
        if mod.__dict__.get("bias") is not None or "bias" in mod._buffers:
            return False
        out.append(0)
        return True
    if (type(p) is not _Parameter or p.dtype is not _BF16 or p.shape != shape[:1] or not p.is_contiguous()
            or p.get_device() != device):
        return False
    at = p.data_ptr()
    if at & 15 or not at:
        return False
    out.append(at)
    return True


def _block(layer, h: int, device: int, out: list):
    """Appends the pointers of one block's tensors, in the order of ``Block`` in the native source, without the cache;
    returns its shape and options, or ``None`` when the block needs the general path.  ``device``: index of the device
    (-1: the CPU) of the hidden states, whose width is ``h``."""
    if type(layer) is not transformer.ParallelTransformerLayer or not layer.plain_block:
        return None
    m = layer._modules
    attn, mlp, n1, n2 = m["attn"], m["mlp"], m["norm1"], m["norm2"]
    gated = type(mlp) is L.ParallelGatedMlp
    if type(attn) is not L.ParallelMHA or type(n1) is not type(n2) or type(n1) not in (L.LayerNorm, L.RMSNorm):
        return None
    if gated:
        if mlp.gate_act is not None:
            return None
    elif type(mlp) is not L.ParallelMLP or not mlp.fused_gelu:
        return None
    if layer.hidden_dropout > 0 and layer.training:
        return None
    am, mm = attn._modules, mlp._modules
    wqkv, wo, w1, w2 = am["Wqkv"], am["out_proj"], mm["fc1"], mm["fc2"]
    for mod in (layer, attn, mlp, n1, n2, wqkv, wo, w1, w2):
        # a forward set on the instance is how adapters and quantisers wrap a layer
        own = mod.__dict__
        if own["_forward_hooks"] or own["_forward_pre_hooks"] or "forward" in own:
            return None
    if (type(wqkv) is not L.ColumnParallelLinear or type(w1) is not L.ColumnParallelLinear
            or type(wo) is not L.RowParallelLinear or type(w2) is not L.RowParallelLinear):
        return None
    if attn.rotary_interleaved or attn.rotary_scale_base is not None or n1.eps != n2.eps:
        return None
    hq, hk, d = attn.local_heads, attn.local_heads_kv, attn.head_dim
    w = w2._parameters.get("weight")
    if w is None or w.dim() != 2:
        return None
    f = w.shape[1]
    for mod, shape in ((n1, (h,)), (wqkv, ((hq + 2 * hk) * d, h)), (wo, (h, hq * d)), (n2, (h,)),
                       (w1, (2 * f if gated else f, h)), (w2, (h, f))):
        if not _tensors(mod, shape, device, out):
            return None
    return hq, hk, d, f, gated, type(n1) is L.RMSNorm, n1.eps, attn.rotary_emb_dim, attn.rotary_emb_base


def _stack(layers, hidden, residual):
    """What the native step takes, for a stack that it covers: the options of its blocks, the addresses of their
    tensors (12 a block), their caches, softmax scales and the parameters of the generation; otherwise ``None``."""
    b, s, h = hidden.shape
    if s != 1 or b > 128 or h % 8 or h > 8192 or not len(layers):
        return None
    if nn_module._global_forward_hooks or nn_module._global_forward_pre_hooks:
        return None
    if Settings.gemm_backend != "tcgen05" or Settings.gemm_max_ctas:       # the step's GEMMs know no limit
        return None
    if residual is not None and (residual.dtype is not _BF16 or residual.shape != hidden.shape
                                 or residual.device != hidden.device):
        return None
    device = hidden.get_device()
    ptrs, scales, ip, kind = [], [], None, None
    for layer in layers:
        k = _block(layer, h, device, ptrs)
        if k is None or (kind is not None and k != kind):
            return None
        attn = layer._modules["attn"]
        mine = attn.__dict__.get("inference_params")
        if mine is None or (ip is not None and mine is not ip):
            return None
        ip, kind = mine, k
        scales.append(attn.softmax_scale)
    hq, hk, d, f, _, _, _, rot, _ = kind
    off = ip.seqlen_offset
    if d % 8 or d > 256 or rot % 16 or f % 64 or hq % hk or off >= ip.max_seqlen:
        return None
    caches = [ip.cache_for(layer._modules["attn"].layer_idx, b, hk, d, hidden.dtype, hidden.device) for layer in layers]
    strides = (caches[0].stride(0), 2 * hk * d, hk * d, d, 1)
    for c in caches:
        if (c.dtype is not _BF16 or c.stride() != strides or c.get_device() != device or c.shape[0] < b
                or c.shape[1] <= off or c.data_ptr() & 15):
            return None
    return kind, ptrs, caches, scales, ip


def _rows(x):
    """``x`` contiguous and on a 16-byte boundary."""
    x = x.contiguous()
    return x.clone() if x.data_ptr() & 15 else x


def stack_step(layers, hidden, residual):
    """``(hidden, residual)`` behind ``layers`` for one new token per sequence (``hidden`` ``[b, 1, h]``), with the
    caches of the blocks' ``inference_params`` extended by it; ``None`` when the general path is needed."""
    if not hidden.is_cuda or hidden.dtype is not _BF16 or torch.is_grad_enabled():
        return None
    found = _stack(layers, hidden, residual)
    if found is None:
        return None
    (hq, hk, d, f, gated, rms, eps, rot, base), ptrs, caches, scales, ip = found
    b, _, h = hidden.shape
    off, cache_sb = ip.seqlen_offset, caches[0].stride(0)
    n = len(caches)
    table = (ctypes.c_uint64 * (_PER_BLOCK * n))()
    for i, c in enumerate(caches):
        table[_PER_BLOCK * i: _PER_BLOCK * (i + 1)] = ptrs[12 * i: 12 * (i + 1)] + [c.data_ptr()]
    cos = sin = 0
    if rot:
        tc, ts = rope_tables(ip.max_seqlen, rot, base, hidden.device)
        cos, sin = tc.data_ptr() + off * rot * 2, ts.data_ptr() + off * rot * 2      # [position][rot / 2] fp32
    hidden, residual = _rows(hidden), None if residual is None else _rows(residual)
    lib = native.kernels()
    x, r = torch.empty_like(hidden), torch.empty_like(hidden)
    scratch = torch.empty(lib.mb_decode_stack_scratch(b, h, hq, hk, d, f), dtype=_BF16, device=hidden.device)
    rc = lib.mb_decode_stack(ptr(hidden), ptr(residual), ptr(x), ptr(r), table, n, ptr(scratch), b, h, hq, hk, d, f,
                             128 if gated else 2, int(rms), float(eps), (ctypes.c_float * n)(*scales), cos, sin, rot,
                             off, cache_sb, stream())
    if rc < 0:
        raise RuntimeError(f"mb_decode_stack failed with code {rc}")
    native.launch_count += rc
    return x, r
