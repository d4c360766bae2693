"""Which kernel a GEMM goes to, with the library replaced by a recorder."""
import pytest
import torch

from mist_b200.ops import functional as F
from mist_b200.ops import native


class _Library:
    def __init__(self):
        self.calls = []

    def __getattr__(self, name):
        def entry(*args):
            self.calls.append((name, args))
            return 0
        return entry


def _route(monkeypatch, m, n, k, **settings):
    lib = _Library()
    monkeypatch.setattr(native, "kernels", lambda: lib)
    monkeypatch.setattr(F, "stream", lambda: 0)
    F._pair_workspace.cache_clear()
    for name, value in settings.items():
        monkeypatch.setattr(F.Settings, name, value)
    try:
        F.gemm(torch.zeros(m, k, dtype=torch.bfloat16), torch.zeros(n, k, dtype=torch.bfloat16))
    finally:
        F._pair_workspace.cache_clear()
    return lib.calls[-1]


# a limit on the CTAs leaves SMs to a kernel that runs beside the GEMM: only kernels that honour it are taken
@pytest.mark.parametrize("m", [1, 16, 128, 129])
def test_cta_limit_is_honoured(m, monkeypatch):
    name, args = _route(monkeypatch, m, 256, 512, gemm_max_ctas=100)
    assert name in ("mb_gemm_pair_split_bf16", "mb_gemm_bf16") and 100 in args


def test_few_tokens_without_a_limit(monkeypatch):
    assert _route(monkeypatch, 1, 4096, 4096)[0] == "mb_gemm_skinny_bf16"
