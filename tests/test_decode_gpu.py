"""Kernels of single-token decoding against fp32 references: split positions, grouped heads, cache append."""
import pytest
import torch

from mist_b200.ops import functional as F

pytestmark = pytest.mark.gpu
DEV = "cuda"


def _rel(a, b):
    return ((a.float() - b).norm() / b.norm()).item()


# around the number of positions at which another CTA joins (64 per CTA) and at ragged tails, with one, two and
# four query heads per CTA; every head-size class (8, 16 and 32 lanes per position)
@pytest.mark.parametrize("nh,nkv,d", [(4, 4, 64), (6, 3, 80), (8, 2, 128), (3, 1, 96), (8, 2, 256)])
@pytest.mark.parametrize("seq_len", [1, 31, 63, 64, 65, 511, 513])
def test_decode_attention_splits(nh, nkv, d, seq_len):
    torch.manual_seed(seq_len)
    b, rows = 2, 520
    cache = torch.randn(b, rows, 2, nkv, d, device=DEV, dtype=torch.bfloat16)
    q = torch.randn(b, (nh + 2 * nkv) * d, device=DEV, dtype=torch.bfloat16)[:, : nh * d].view(b, nh, d)
    out = F.decode_attention(q, cache[:, :, 0], cache[:, :, 1], seq_len)
    ref = F.decode_attention(q.cpu().float(), cache[:, :, 0].cpu().float(), cache[:, :, 1].cpu().float(), seq_len)
    # fp32 sums, one rounding of the result to bf16: at most 2^-9 of a value, 2^-10.8 rms
    assert _rel(out.cpu(), ref) < 2 ** -9


@pytest.mark.parametrize("hq,hk,d,rot,s", [(4, 4, 64, 64, 1), (8, 2, 128, 32, 7), (4, 4, 80, 16, 33), (6, 3, 80, 0, 5)])
def test_rope_append(hq, hk, d, rot, s):
    torch.manual_seed(s)
    b, rows, off = 3, 50, 9
    qkv = torch.randn(b, s, (hq + 2 * hk) * d, device=DEV, dtype=torch.bfloat16)
    cache = torch.full((b + 1, rows, 2, hk, d), 7.0, device=DEV, dtype=torch.bfloat16)
    rotary = None
    want = qkv[..., : (hq + hk) * d].reshape(b, s, 1, hq + hk, d).cpu()
    if rot:
        cos, sin = F.rope_tables(rows, rot, 10000.0, DEV)
        rotary = (cos[off:off + s], sin[off:off + s], rot)
        want = F._rope_apply(want, rotary[0].cpu(), rotary[1].cpu(), rot, False, 1)
    want = want.view(b, s, hq + hk, d)
    v = qkv[..., (hq + hk) * d:].view(b, s, hk, d).clone()
    F.rope_append_(qkv, cache, off, hq, hk, d, rotary)
    ulp = dict(atol=1e-6, rtol=2 ** -7)       # one bf16 rounding either way
    torch.testing.assert_close(qkv[..., : hq * d].view(b, s, hq, d).cpu(), want[:, :, :hq], **ulp)
    torch.testing.assert_close(cache[:b, off:off + s, 0].cpu(), want[:, :, hq:], **ulp)
    assert torch.equal(cache[:b, off:off + s, 1], v)
    keep = torch.ones(rows, dtype=torch.bool)
    keep[off:off + s] = False
    assert (cache[:b, keep.to(DEV)] == 7).all() and (cache[b] == 7).all()


# M: the sides of every token-tile size (16, 32, 64, 128); N: one tile, a tail of one column pair and of an odd
# column; K: one k-block, a K tail, and enough for two, four and eight CTAs per tile
@pytest.mark.parametrize("M", [1, 16, 17, 33, 64, 65, 128])
@pytest.mark.parametrize("N,K", [(128, 64), (130, 72), (333, 1024), (384, 2056), (256, 4096)])
def test_skinny_gemm(M, N, K):
    torch.manual_seed(M)
    x = torch.randn(M, K, device=DEV, dtype=torch.bfloat16)
    w = torch.randn(N, K, device=DEV, dtype=torch.bfloat16) * K ** -0.5
    bias = torch.randn(N, device=DEV, dtype=torch.bfloat16)
    res = torch.randn(M, N, device=DEV, dtype=torch.bfloat16)
    ref = x.float() @ w.float().t()
    # fp32 sums and one rounding to bf16 (2^-9 of a value at most); GELU adds the 2^-11 of its tanh
    assert _rel(F.gemm(x, w), ref) < 2 ** -9
    assert _rel(F.gemm(x, w, bias=bias, aux=res, flags=F.EPI_RESIDUAL), ref + bias.float() + res.float()) < 2 ** -9
    act = torch.nn.functional.gelu(ref + bias.float(), approximate="tanh")
    assert _rel(F.gemm(x, w, bias=bias, flags=F.EPI_GELU), act) < 2 ** -8
