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
    (2, 32, 64, 64, 64, 64, False),        # the largest problem of the one-block backward kernel, and past it on each side
    (2, 33, 64, 8, 8, 64, False),
    (2, 32, 65, 8, 8, 128, True),
    (3, 20, 20, 43, 43, 80, True),
    (2, 20, 20, 8, 4, 96, True),
    (2, 127, 127, 2, 2, 64, True),         # one short of a tile
    (1, 129, 129, 2, 1, 80, True),         # one row in the second tile
    (1, 257, 257, 4, 2, 96, True),         # one row in a second pair of tiles
    (2, 200, 513, 2, 2, 128, True),        # fewer queries than keys
    (1, 640, 300, 2, 2, 128, True),        # queries that see no key
    (1, 384, 384, 3, 3, 112, False),
    (3, 640, 640, 40, 10, 80, True),       # more work items than CTAs, dQ beside dV and dK in tensor memory
    (2, 1024, 1024, 24, 4, 128, True),     # the same, dQ over dP
    # both sides of the sizes at which the forward kernel of one tile per CTA takes over
    (2, 64, 64, 3, 3, 64, True),
    (2, 65, 64, 3, 3, 64, False),
    (2, 32, 64, 4, 2, 128, True),
    (2, 33, 64, 4, 2, 128, True),
    (149, 32, 1024, 1, 1, 48, True),       # more heads than SMs: fewer queries than keys
    (37, 64, 320, 4, 2, 64, False),
    (37, 64, 100, 4, 4, 32, True),         # queries and keys of less than a tile, three key blocks of 64
    (10, 128, 150, 15, 5, 32, True),
    (75, 64, 64, 2, 2, 128, False),
    (1, 192, 192, 4, 4, 64, True),         # two tiles, each on a CTA of its own
    (1, 300, 64, 4, 4, 64, True),          # queries that see no key
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


# s, heads, kv heads, lengths: own heads; groups summed after the kernel, and inside it; short sequences
@pytest.mark.parametrize("s,nh,nkv,lens", [(400, 6, 6, [400, 1, 128, 257]), (400, 6, 2, [400, 1, 128, 257]),
                                           (640, 24, 8, [640, 129, 1, 500, 640, 64, 333, 256]),
                                           (60, 6, 3, [60, 1, 33]), (32, 160, 160, [7, 32])])
@pytest.mark.parametrize("causal", [True, False])
@pytest.mark.parametrize("d", [64, 128])
def test_block_kernels_on_padded_batches(s, nh, nkv, lens, d, causal):
    torch.manual_seed(d)
    b = len(lens)
    q, g = (torch.randn(b, s, nh, d, device=DEV, dtype=torch.bfloat16) for _ in range(2))
    k, v = (torch.randn(b, s, nkv, d, device=DEV, dtype=torch.bfloat16) for _ in range(2))
    lens = torch.tensor(lens, device=DEV, dtype=torch.int32)
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


def _rotate(x, cos, sin, rot):
    """The rotation in 64 bits: channels in halves, ``x`` ``[b, s, heads, d]``."""
    c, sn = cos.double()[:, None], sin.double()[:, None]
    x1, x2 = x[..., :rot // 2], x[..., rot // 2:rot]
    return torch.cat([x1 * c - x2 * sn, x1 * sn + x2 * c, x[..., rot:]], -1)


@pytest.mark.parametrize("nh,nkv,d,rot", [(4, 4, 64, 64), (6, 2, 80, 32), (8, 2, 128, 128)])
@pytest.mark.parametrize("lens", [None, [300, 17, 129]])
def test_projection_with_rotary_and_lengths(nh, nkv, d, rot, lens):
    torch.manual_seed(d)
    b, s = 3, 300
    x = torch.randn(b, s, nh + 2 * nkv, d, device=DEV, dtype=torch.bfloat16, requires_grad=True)
    g = torch.randn(b, s, nh, d, device=DEV, dtype=torch.bfloat16)
    lens = None if lens is None else torch.tensor(lens, device=DEV, dtype=torch.int32)
    cos, sin = F.rope_tables(s, rot, 10000.0, DEV)
    scale = 1 / math.sqrt(d)
    o = F.attention_projected(x.clone(), nkv, scale, True, (cos, sin, rot), lens)
    o.backward(g)
    native.check_status()
    leaf = x.detach().double().requires_grad_(True)
    q, k, v = leaf.split([nh, nkv, nkv], 2)
    o_ref, _ = _exact(_rotate(q, cos, sin, rot), _rotate(k, cos, sin, rot), v, scale, True, lens, lens)
    o_ref.backward(g.double())
    # q and k are rounded to bf16 once more, behind the rotation, and so is their gradient: a third and a fourth rounding of
    # 2^-9 each, independent of the two above
    for got, want in zip((o, *x.grad.split([nh, nkv, nkv], 2)), (o_ref, *leaf.grad.split([nh, nkv, nkv], 2))):
        diff = got.double() - want
        assert torch.isfinite(got).all() and diff.norm() <= 2 ** -7.5 * want.norm()
        assert diff.abs().max() <= 2 ** -6 * want.abs().max()


@pytest.mark.parametrize("nh,nkv,d", [(4, 4, 64), (6, 2, 128)])
@pytest.mark.parametrize("sq,sk", [(40, 300), (300, 40)])
@pytest.mark.parametrize("padded", [False, True])
def test_packed_keys_and_values(nh, nkv, d, sq, sk, padded):
    torch.manual_seed(sq)
    b, scale = 2, 0.1
    q = torch.randn(b, sq, nh, d, device=DEV, dtype=torch.bfloat16, requires_grad=True)
    kv = torch.randn(b, sk, 2, nkv, d, device=DEV, dtype=torch.bfloat16, requires_grad=True)
    g = torch.randn(b, sq, nh, d, device=DEV, dtype=torch.bfloat16)
    lens_q, lens_k = (torch.tensor([n, n // 3], device=DEV, dtype=torch.int32) if padded else None for n in (sq, sk))
    o = F.attention_kvpacked(q, kv, scale, False, lens_q, lens_k)
    o.backward(g)
    native.check_status()
    q_ref, kv_ref = (t.detach().double().requires_grad_(True) for t in (q, kv))
    o_ref, _ = _exact(q_ref, kv_ref[:, :, 0], kv_ref[:, :, 1], scale, False, lens_q, lens_k)
    o_ref.backward(g.double())
    for got, want in ((o, o_ref), (q.grad, q_ref.grad), (kv.grad, kv_ref.grad)):
        _close(got, want)
