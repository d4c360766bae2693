"""The attention kernels on 128 x 128 blocks (two query tiles per CTA forward; persistent backward) at the edges of their
tiles, against attention in 64 bits on the same bf16 inputs.

Bounds: probabilities (and dS) are rounded to bf16 before a product with fp32 accumulation, results to bf16 once more: two
roundings of at most 2^-9 each, independent from term to term, so 2^-8 of the norm holds with room; single values may be
sums of few terms, where both roundings are seen in full (2^-7 of the largest value)."""
import math

import pytest
import torch

from mist_b200.ops import attention_bwd, native
from mist_b200.ops import functional as F

pytestmark = pytest.mark.gpu
DEV = "cuda"


def _exact(q, k, v, scale, causal, lens_q=None, lens_k=None):
    b, sq, nh, _ = q.shape
    sk, g = k.shape[1], nh // k.shape[2]
    k, v = k.repeat_interleave(g, 2), v.repeat_interleave(g, 2)
    s = torch.einsum("bqhd,bkhd->bhqk", q, k) * scale
    lq = torch.full((b,), sq, device=DEV) if lens_q is None else lens_q.long()
    lk = torch.full((b,), sk, device=DEV) if lens_k is None else lens_k.long()
    i, j = torch.arange(sq, device=DEV)[:, None], torch.arange(sk, device=DEV)[None]
    see = (i < lq[:, None, None]) & (j < lk[:, None, None])
    if causal:
        see = see & (j <= i + (lk - lq)[:, None, None])
    see = see[:, None]
    s = s.masked_fill(~see, -math.inf)
    seen = see.any(-1, keepdim=True)
    p = torch.where(seen, torch.softmax(torch.where(seen, s, torch.zeros_like(s)), -1), torch.zeros_like(s))
    return torch.einsum("bhqk,bkhd->bqhd", p, v), torch.logsumexp(s, -1)


def _close(got, want):
    want = want.double()
    diff = got.double() - want
    assert torch.isfinite(got).all()
    assert diff.norm() <= 2 ** -8 * want.norm() + 1e-6
    assert diff.abs().max() <= 2 ** -7 * want.abs().max() + 1e-6


SHAPES = [  # b, sq, sk, heads, kv heads, d, causal
    (1, 1, 1, 1, 1, 16, True),             # one row
    (2, 127, 127, 2, 2, 64, True),         # one short of a tile
    (1, 129, 129, 2, 1, 80, True),         # one row in the second tile
    (1, 257, 257, 4, 2, 96, True),         # one row in a second pair of tiles
    (2, 200, 513, 2, 2, 128, True),        # fewer queries than keys
    (1, 640, 300, 2, 2, 128, True),        # queries that see no key
    (1, 384, 384, 3, 3, 112, False),
    (3, 640, 640, 40, 10, 80, True),       # more work items than CTAs, dQ beside dV and dK in tensor memory
    (2, 1024, 1024, 24, 4, 128, True),     # the same, dQ over dP
]


@pytest.mark.parametrize("b,sq,sk,nh,nkv,d,causal", SHAPES)
def test_block_kernels_at_tile_edges(b, sq, sk, nh, nkv, d, causal):
    torch.manual_seed(b * sq + d)
    q, g = (torch.randn(b, sq, nh, d, device=DEV, dtype=torch.bfloat16) for _ in range(2))
    k, v = (torch.randn(b, sk, nkv, d, device=DEV, dtype=torch.bfloat16) for _ in range(2))
    scale = 1 / math.sqrt(d)
    leaves = [t.double().requires_grad_(True) for t in (q, k, v)]
    o_ref, lse_ref = _exact(*leaves, scale, causal)
    o, lse = F.attn_fwd(q, k, v, scale, causal)
    _close(o, o_ref)
    seen = torch.isfinite(lse_ref)
    assert torch.equal(torch.isfinite(lse), seen)
    # scores are sums of d fp32 terms, the logarithm of a sum of fp32 exponentials
    assert (lse[seen].double() - lse_ref[seen]).abs().max() < 1e-4
    grads = attention_bwd.backward(g, q, k, v, o, lse, scale, causal)
    native.check_status()
    for got, want in zip(grads, torch.autograd.grad(o_ref, leaves, g.double())):
        _close(got, want)


@pytest.mark.parametrize("causal", [True, False])
@pytest.mark.parametrize("d", [64, 128])
def test_block_kernels_on_padded_batches(d, causal):
    torch.manual_seed(d)
    b, s, nh = 4, 400, 6
    q, k, v, g = (torch.randn(b, s, nh, d, device=DEV, dtype=torch.bfloat16) for _ in range(4))
    lens = torch.tensor([400, 1, 128, 257], device=DEV, dtype=torch.int32)
    scale = 1 / math.sqrt(d)
    leaves = [t.double().requires_grad_(True) for t in (q, k, v)]
    o_ref, _ = _exact(*leaves, scale, causal, lens, lens)
    o, lse = F.attn_fwd(q, k, v, scale, causal, seqlens_q=lens, seqlens_k=lens)
    _close(o, o_ref)
    grads = attention_bwd.backward(g, q, k, v, o, lse, scale, causal, seqlens=(lens, lens))
    native.check_status()
    for got, want in zip(grads, torch.autograd.grad(o_ref, leaves, g.double())):
        _close(got, want)


@pytest.mark.parametrize("nh,nkv,s", [(8, 2, 300), (4, 4, 257), (16, 4, 2048)])
def test_gradients_into_a_packed_projection(nh, nkv, s):
    """dK and dV of a group, summed over parts or in the CTA, land in strided views of one gradient."""
    torch.manual_seed(s)
    b, d, scale = 2, 80, 0.11
    qkv = torch.randn(b, s, nh + 2 * nkv, d, device=DEV, dtype=torch.bfloat16, requires_grad=True)
    g = torch.randn(b, s, nh, d, device=DEV, dtype=torch.bfloat16)
    o = F.attention_projected(qkv, nkv, scale, True)
    o.backward(g)
    native.check_status()
    leaf = qkv.detach().double().requires_grad_(True)
    o_ref, _ = _exact(*leaf.split([nh, nkv, nkv], 2), scale, True)
    o_ref.backward(g.double())
    _close(o, o_ref)
    for got, want in zip(qkv.grad.split([nh, nkv, nkv], 2), leaf.grad.split([nh, nkv, nkv], 2)):
        _close(got, want)
