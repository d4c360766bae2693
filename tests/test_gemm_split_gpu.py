"""The CTA-pair GEMM with the tiles of its last wave cut along K, against 64 bits.

Bounds: a bf16 result is rounded once (2^-9 of each value at most, 2^-8 allows for GELU's approximation beside it); an fp32
result carries the error of the tensor core's fp32 sums, which grows with the number of terms: 1.86e-5 of the norm for an
unsplit sum of 16384, the longest here, and less in parts.  2e-5 allows that."""
import pytest
import torch

from mist_b200.ops import functional as F
from mist_b200.ops import native

pytestmark = pytest.mark.gpu
DEV = "cuda"


# M, N, K, a_mn, b_mn: two parts, three with a ragged K, four; ragged M and N (the second CTA of a pair past the bottom)
@pytest.mark.parametrize("M,N,K,a_mn,b_mn", [(2560, 2560, 16384, True, True), (5632, 1024, 7000, True, True),
                                             (4864, 1024, 16384, True, False),
                                             (2440, 2600, 8200, True, True), (2304, 2560, 8192, False, False),
                                             (2440, 2600, 8200, False, True)])
@pytest.mark.parametrize("form", ["bf16", "accumulate", "bias_gelu_pre"])
def test_split_tiles(M, N, K, a_mn, b_mn, form):
    torch.manual_seed(K)
    flags = {"bf16": 0, "accumulate": F.EPI_ACCUM, "bias_gelu_pre": F.EPI_GELU | F.EPI_SAVE_PRE}[form]
    fp32 = F.EPI_OUT_FP32 if form == "accumulate" else 0
    bias_flag = F.EPI_BIAS if form == "bias_gelu_pre" else 0
    assert native.kernels().mb_gemm_pair_workspace(M, N, K, flags | fp32 | bias_flag, 0) > 0
    a = torch.randn(*((K, M) if a_mn else (M, K)), device=DEV, dtype=torch.bfloat16)
    b = torch.randn(*((K, N) if b_mn else (N, K)), device=DEV, dtype=torch.bfloat16) * K ** -0.5
    want = (a.double().t() if a_mn else a.double()) @ (b.double() if b_mn else b.double().t())
    if form == "accumulate":
        out = torch.ones(M, N, device=DEV)
        F.gemm(a, b, a_mn=a_mn, b_mn=b_mn, out=out, flags=flags)
        assert (out - want - 1).norm() < 2e-5 * want.norm()
    elif form == "bf16":
        out = F.gemm(a, b, a_mn=a_mn, b_mn=b_mn)
        assert (out - want).norm() < 2 ** -8 * want.norm()
        assert torch.equal(out, F.gemm(a, b, a_mn=a_mn, b_mn=b_mn))        # parts are added in K order
    else:
        bias, pre = torch.randn(N, device=DEV, dtype=torch.bfloat16), torch.empty(M, N, device=DEV, dtype=torch.bfloat16)
        out = F.gemm(a, b, a_mn=a_mn, b_mn=b_mn, bias=bias, aux=pre, flags=flags)
        want = want + bias.double()
        assert (pre - want).norm() < 2 ** -8 * want.norm()
        want = torch.nn.functional.gelu(want, approximate="tanh")
        assert (out - want).norm() < 2 ** -8 * want.norm()
    native.check_status()
