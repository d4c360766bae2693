"""The packed attention paths rotate in place only what nobody else holds: the output of a projection that has a hook, or
that was replaced, stays as it was, and need not be contiguous."""
import pytest
import torch

from mist_b200.inference import InferenceParams
from mist_b200.modules.layers import PaddingMask, ParallelMHA


def _layer(kv_heads, rot, device, dtype):
    torch.manual_seed(0)
    m = ParallelMHA(256, 4, kv_heads, causal=True, rotary_emb_dim=rot, layer_idx=0, device=device, dtype=dtype)
    for p in m.parameters():
        torch.nn.init.normal_(p, std=0.1)
    return m


def _mask(device):
    return PaddingMask(torch.arange(9, device=device)[None] < torch.tensor([[9], [4]], device=device))


def _strided_forward(m):
    own = m.Wqkv.forward

    def forward(x):
        y = own(x)
        return torch.cat([y, y], -1)[..., :y.shape[-1]]
    return forward


def _check_strided(kv_heads, rot, masked, device, dtype):
    m = _layer(kv_heads, rot, device, dtype)
    x = torch.randn(2, 9, 256, device=device, dtype=dtype)
    mask = _mask(device) if masked else None
    want = m(x, attention_mask=mask)
    m.Wqkv.forward = _strided_forward(m)
    torch.testing.assert_close(m(x, attention_mask=mask), want)


@pytest.mark.parametrize("rot", [0, 32])
@pytest.mark.parametrize("masked", [False, True])
def test_strided_projection_cpu(rot, masked):
    _check_strided(2, rot, masked, "cpu", torch.float32)


@pytest.mark.gpu
@pytest.mark.parametrize("rot", [0, 32])
@pytest.mark.parametrize("masked", [False, True])
def test_strided_projection_gpu(rot, masked):
    _check_strided(2, rot, masked, "cuda", torch.bfloat16)


@pytest.mark.gpu
@pytest.mark.parametrize("kv_heads,masked", [(2, False), (2, True), (4, True)])
@pytest.mark.parametrize("cached", [False, True])
def test_hooked_projection_keeps_its_output(kv_heads, masked, cached):
    if cached and masked:
        pytest.skip("a cached prompt has no mask")
    m = _layer(kv_heads, 32, "cuda", torch.bfloat16)
    x = torch.randn(2, 9, 256, device="cuda", dtype=torch.bfloat16)
    with torch.no_grad():
        want = m.Wqkv(x)
        seen = []
        m.Wqkv.register_forward_hook(lambda mod, args, out: seen.append(out))
        m.inference_params = InferenceParams(2, 12) if cached else None
        plain = m(x) if cached else m(x, attention_mask=_mask("cuda") if masked else None)
    assert torch.equal(seen[0], want) and bool(plain.isfinite().all())
