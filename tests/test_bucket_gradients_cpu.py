"""Weight gradients go into the flat bucket also from a block that is recomputed in the backward pass, where the saved
weight comes back as another tensor."""
import pytest
import torch
from torch.utils.checkpoint import checkpoint

from mist_b200.ops import functional as F


@pytest.mark.parametrize("recompute", [False, True])
@pytest.mark.parametrize("accumulate", [False, True])
def test_linear_writes_its_bucket(recompute, accumulate):
    torch.manual_seed(0)
    w = torch.nn.Parameter(torch.randn(5, 8))
    x, g = torch.randn(3, 8, requires_grad=True), torch.randn(3, 5)
    w.grad_bucket, w.grad_accumulate = torch.ones(5, 8), accumulate
    y = checkpoint(F.linear, x, w, use_reentrant=False) if recompute else F.linear(x, w)
    y.backward(g)
    assert w.grad is None and w.grad_accumulate
    torch.testing.assert_close(w.grad_bucket, g.t() @ x.detach() + (1.0 if accumulate else 0.0))
    torch.testing.assert_close(x.grad, g @ w.detach())
