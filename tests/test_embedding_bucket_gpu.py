"""Embedding gradients summed into the flat bucket, against an fp32 scatter.

The fp32 sums differ by the order of the atomics (2^-22 of values of a few units here); a bf16 bucket is rounded once."""
import pytest
import torch

from mist_b200.ops import functional as F
from mist_b200.ops import native

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16, torch.float16, torch.float64])
@pytest.mark.parametrize("accumulate", [False, True])
@pytest.mark.parametrize("offset", [0, 2])          # elements before the bucket: 16-byte accesses need aligned rows
@pytest.mark.parametrize("strided", [False, True])  # rows of a wider buffer
def test_embedding_bucket(dtype, accumulate, offset, strided):
    torch.manual_seed(1)
    v, h, start = 37, 24, 5
    w = torch.nn.Parameter(torch.randn(v, h, device=DEV, dtype=torch.bfloat16))
    ids = torch.randint(0, v + 2 * start, (3, 50), device=DEV)          # some outside this rank's slice
    g = torch.randn(3, 50, h, device=DEV, dtype=torch.bfloat16)
    wide = h + 8 if strided else h
    flat = torch.randn(offset + v * wide, device=DEV).to(dtype)
    bucket, before = flat[offset:].view(v, wide)[:, :h], flat.clone()
    old = bucket.double().clone() if accumulate else torch.zeros(v, h, device=DEV, dtype=torch.double)
    w.grad_bucket, w.grad_accumulate = bucket, accumulate
    F.embedding(ids, w, None, start).backward(g)
    native.check_status()
    inside = ((ids >= start) & (ids < start + v)).reshape(-1)
    want = old.index_add(0, (ids.reshape(-1) - start)[inside], g.double().reshape(-1, h)[inside])
    assert w.grad is None and w.grad_accumulate
    # fp32 sums (2^-20); one rounding of a narrower bucket: 2^-8 of a value in bf16, 2^-10 in fp16
    bound = {torch.bfloat16: 2 ** -8, torch.float16: 2 ** -10}.get(dtype, 2 ** -20)
    assert ((bucket.double() - want).abs() <= bound * want.abs().clamp(min=1.0)).all()
    outside = torch.ones(flat.numel(), dtype=torch.bool, device=DEV)
    outside[offset:].view(v, wide)[:, :h] = False
    assert torch.equal(flat[outside], before[outside])
