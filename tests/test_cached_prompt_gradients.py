"""Gradients through a prompt that fills the key/value cache are those of the same attention without a cache."""
import pytest
import torch

from mist_b200.inference import InferenceParams
from mist_b200.modules.layers import ParallelMHA


def _check(device, dtype, kv_heads, rot):
    torch.manual_seed(0)
    m = ParallelMHA(256, 4, kv_heads, causal=True, rotary_emb_dim=rot, layer_idx=0, device=device, dtype=dtype)
    for p in m.parameters():
        torch.nn.init.normal_(p, std=0.1)
    x, g = (torch.randn(2, 9, 256, device=device, dtype=dtype) for _ in range(2))
    grads = []
    for ip in (None, InferenceParams(2, 12)):
        m.inference_params = ip
        m.zero_grad()
        leaf = x.clone().requires_grad_(True)
        m(leaf).backward(g)
        grads.append([leaf.grad.float()] + [p.grad.float() for p in m.parameters()])
    # one precision throughout: sums in another order, and in bf16 a rounding of each value on the way (2^-9, a few)
    bound = 1e-5 if dtype == torch.float32 else 2e-2
    for a, r in zip(*grads[::-1]):
        assert (a - r).norm() <= bound * r.norm()


@pytest.mark.parametrize("kv_heads", [4, 2])
@pytest.mark.parametrize("rot", [0, 32])
def test_cached_prompt_cpu(kv_heads, rot):
    _check("cpu", torch.float32, kv_heads, rot)


@pytest.mark.gpu
@pytest.mark.parametrize("kv_heads", [4, 2])
@pytest.mark.parametrize("rot", [0, 32])
def test_cached_prompt_gpu(kv_heads, rot):
    _check("cuda", torch.bfloat16, kv_heads, rot)
