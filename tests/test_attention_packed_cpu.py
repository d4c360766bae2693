"""Attention over a packed projection output gives what splitting it, rotating out of place and attending gives, and the
gradient of the packed tensor is that of the parts."""
import pytest
import torch

from mist_b200.modules import layers
from mist_b200.ops import functional as F


def _layer(heads, kv_heads, rot, causal, cross=False):
    torch.manual_seed(0)
    m = layers.ParallelMHA(heads * 16, heads, kv_heads, causal=causal, rotary_emb_dim=rot, cross_attn=cross)
    for p in m.parameters():
        torch.nn.init.normal_(p, std=0.1)
    return m


def _split_forward(m, x, mask, kv=None, kv_mask=None):
    b, s, _ = x.shape
    hq, hk, d = m.local_heads, m.local_heads_kv, m.head_dim
    if kv is not None:
        q = m.Wq(x).view(b, s, hq, d)
        k, v = m.Wkv(kv).view(b, kv.shape[1], 2, hk, d).unbind(2)
    else:
        q, k, v = m.Wqkv(x).view(b, s, hq + 2 * hk, d).split([hq, hk, hk], 2)
        if m.rotary_emb_dim:
            cos, sin = F.rope_tables(s, m.rotary_emb_dim, m.rotary_emb_base, x.device)
            qk = layers._RotaryOutOfPlace.apply(torch.cat([q, k], 2).unsqueeze(2), cos, sin, m.rotary_emb_dim, 1)
            q, k = qk.squeeze(2).split([hq, hk], 2)
        kv_mask = mask
    o = F.attention(q, k, v, m.softmax_scale, m.causal, None if mask is None else mask.lengths_dev,
                    None if kv_mask is None else kv_mask.lengths_dev)
    return m.out_proj(o.reshape(b, s, -1))


def _compare(m, inputs, call, reference):
    outs, grads = [], []
    for f in (call, reference):
        leaves = [t.clone().requires_grad_(True) for t in inputs]
        m.zero_grad()
        y = f(*leaves)
        (y * torch.linspace(-1, 1, y.numel()).view_as(y)).sum().backward()
        outs.append(y)
        grads.append([t.grad for t in leaves] + [p.grad.clone() for p in m.parameters()])
    torch.testing.assert_close(outs[0], outs[1], rtol=1e-5, atol=1e-6)
    for a, b in zip(*grads):
        torch.testing.assert_close(a, b, rtol=1e-4, atol=1e-5)


@pytest.mark.parametrize("heads,kv_heads", [(4, 4), (4, 2), (6, 1)])
@pytest.mark.parametrize("rot", [0, 8, 16])
@pytest.mark.parametrize("causal", [True, False])
@pytest.mark.parametrize("lens", [None, [9, 4, 1]])
def test_self_attention(heads, kv_heads, rot, causal, lens):
    m = _layer(heads, kv_heads, rot, causal)
    x = torch.randn(3, 9, heads * 16)
    mask = None if lens is None else layers.PaddingMask(torch.arange(9)[None] < torch.tensor(lens)[:, None])
    _compare(m, [x], lambda t: m(t, attention_mask=mask), lambda t: _split_forward(m, t, mask))


@pytest.mark.parametrize("kv_heads", [4, 2])
@pytest.mark.parametrize("masked", [False, True])
def test_cross_attention(kv_heads, masked):
    m = _layer(4, kv_heads, 0, False, cross=True)
    x, kv = torch.randn(2, 5, 64), torch.randn(2, 9, 64)
    mask = layers.PaddingMask(torch.arange(5)[None] < torch.tensor([[5], [3]])) if masked else None
    kv_mask = layers.PaddingMask(torch.arange(9)[None] < torch.tensor([[2], [9]])) if masked else None
    _compare(m, [x, kv], lambda a, b: m(a, b, attention_mask=mask, kv_mask=kv_mask),
             lambda a, b: _split_forward(m, a, mask, b, kv_mask))


def test_qkvpacked_takes_strided_input():
    wide = torch.randn(2, 7, 3, 4, 24)
    ref = F.attention(wide[:, :, 0, :, :16], wide[:, :, 1, :, :16], wide[:, :, 2, :, :16])
    torch.testing.assert_close(F.attention_qkvpacked(wide[..., :16]), ref, rtol=1e-6, atol=1e-6)


def test_block_size_settings_are_accepted():
    q, k, v = (torch.randn(1, 5, 2, 16) for _ in range(3))
    want, _ = F.attn_fwd(q, k, v, 0.25, True)
    assert torch.equal(F.attn_fwd(q, k, v, 0.25, True, block_n=F.Settings.attn_block_n)[0], want)
