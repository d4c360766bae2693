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


# both sides of the lengths at which another kernel takes over, for few and for many heads; one stage of the ring, two and
# all of them, and lengths that make two, four and eight CTAs share a sequence
@pytest.mark.parametrize("b,nh,nkv,d", [(1, 2, 2, 64), (10, 32, 32, 64), (2, 6, 3, 40), (3, 8, 2, 128), (33, 16, 4, 80),
                                        (2, 8, 2, 256), (9, 5, 1, 136), (40, 8, 8, 16)])
@pytest.mark.parametrize("seq_len", [1, 12, 13, 16, 17, 32, 33, 40, 41, 96, 97, 129, 200, 257, 600, 1100])
def test_decode_attention_kernels(b, nh, nkv, d, seq_len):
    torch.manual_seed(seq_len)
    cache = torch.randn(b, seq_len + 2, 2, nkv, d, device=DEV, dtype=torch.bfloat16)
    q = torch.randn(b, nh, d, device=DEV, dtype=torch.bfloat16)
    cache[:, seq_len:] = float("nan")                 # what lies behind the last position takes no part
    out = F.decode_attention(q, cache[:, :, 0], cache[:, :, 1], seq_len)
    k, v = (cache[:, :seq_len, i].double().repeat_interleave(nh // nkv, 2) for i in (0, 1))
    p = torch.softmax(torch.einsum("bhd,bkhd->bhk", q.double(), k) / d ** 0.5, -1)
    assert _rel(out, torch.einsum("bhk,bkhd->bhd", p, v)) < 2 ** -9          # one rounding to bf16


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


# The kernel itself, also where another one is faster: K for one to eight CTAs per tile (four K blocks each), a K tail,
# rows of one token, of whole rounds of tokens and one more; C rows that allow 8-byte, 4-byte and 2-byte stores
@pytest.mark.parametrize("M", [1, 6, 16, 17, 33, 65, 128])
@pytest.mark.parametrize("N,K,ldc", [(192, 64, 192), (128, 520, 128), (320, 768, 324), (128, 1024, 130),
                                     (128, 1280, 131), (64, 1536, 64), (128, 1800, 128), (448, 2048, 450)])
@pytest.mark.parametrize("epi", ["plain", "gelu", "residual", "swiglu", "swiglu_bias"])
def test_skinny_kernel(M, N, K, ldc, epi):
    from mist_b200.ops import native
    torch.manual_seed(N + K)
    swiglu = epi.startswith("swiglu")
    rows = 2 * N if swiglu else N
    x = torch.randn(M, K, device=DEV, dtype=torch.bfloat16)
    w = torch.randn(rows, K, device=DEV, dtype=torch.bfloat16) * K ** -0.5
    bias = torch.randn(rows, device=DEV, dtype=torch.bfloat16)
    aux = torch.randn(M, ldc, device=DEV, dtype=torch.bfloat16)
    out = torch.full((M, ldc), 7.0, device=DEV, dtype=torch.bfloat16)
    flags = {"plain": 0, "gelu": F.EPI_BIAS | F.EPI_GELU, "residual": F.EPI_RESIDUAL, "swiglu": 128,
             "swiglu_bias": 128 | F.EPI_BIAS}[epi]
    native.call("mb_gemm_skinny_bf16", x.data_ptr(), w.data_ptr(), out.data_ptr(), M, N, K, K, K, ldc, flags,
                bias.data_ptr(), aux.data_ptr(), 1.0, 1, 0, native.stream())
    ref = x.double() @ w.double().t() + (bias.double() if flags & F.EPI_BIAS else 0)
    if epi == "gelu":
        ref = torch.nn.functional.gelu(ref, approximate="tanh")
    elif epi == "residual":
        ref = ref + aux[:, :N].double()
    elif swiglu:
        ref = torch.nn.functional.silu(ref[:, :N]) * ref[:, N:]
    # fp32 sums and one rounding to bf16 (2^-9 of a value at most); the activations add the error of their exponential
    # (2^-11)
    assert _rel(out[:, :N], ref) < (2 ** -9 if epi in ("plain", "residual") else 2 ** -8)
    assert (out[:, N:] == 7).all()


@pytest.mark.parametrize("model,extra", [("gpt2/1.3b", []), ("llama/1.3b", []), ("llama/1.3b", ["model.num_heads_kv=2"])])
@pytest.mark.parametrize("b", [1, 5, 40])
def test_native_decode_step_matches_the_modules(model, extra, b, monkeypatch):
    """The whole stack in one call against the same step through the modules, over several tokens."""
    from mist_b200.config import load_config
    from mist_b200.inference import kv_cache
    from mist_b200.models.provider import base_model_provider
    from mist_b200.ops import decode
    cfg, _ = load_config("config", ["experiment=gpt2-1.3b", f"model={model}", "model.num_hidden_layers=3",
                                    "model.hidden_size=512", "model.intermediate_size=1408",
                                    "model.num_attention_heads=8", "model.vocab_size=1024",
                                    "training.max_sequence_length=64", "strategy.layer_partitions=[3]"] + extra,
                         check_world_size=False)
    torch.manual_seed(0)
    net = base_model_provider(cfg.model, device=torch.device(DEV), dtype=torch.bfloat16).eval()
    ids = torch.randint(0, 1024, (b, 12), device=DEV)

    def steps():
        out = []
        with torch.no_grad(), kv_cache(net, b, 16) as ip:
            for t in range(12):
                pos = torch.full((b, 1), t, device=DEV)
                out.append(net(ids[:, t:t + 1], position_ids=pos).reshape(b, -1).float())
                ip.seqlen_offset += 1
            return torch.stack(out), [ip.key_value_memory[i].float() for i in range(3)]

    calls = []
    native_step = decode.stack_step
    monkeypatch.setattr(decode, "stack_step", lambda *a: calls.append(native_step(*a)) or calls[-1])
    got, cache = steps()
    assert len(calls) == 12 and all(c is not None for c in calls)
    monkeypatch.setattr(decode, "stack_step", lambda *a: None)
    want, cache_ref = steps()
    # three blocks of bf16 roundings at different places (SwiGLU takes unrounded products here)
    assert _rel(got, want) < 2e-2
    for a, r in zip(cache, cache_ref):
        assert _rel(a, r) < 2e-2


# batches of every token-tile size, the largest that the step takes, and a residual stream that comes in
@pytest.mark.parametrize("model", ["gpt2/1.3b", "llama/1.3b"])
@pytest.mark.parametrize("b,with_residual", [(3, True), (20, False), (65, True), (128, False)])
def test_native_decode_step_takes_every_parameter(model, b, with_residual, monkeypatch):
    """Biases on every linear and no two norms alike: each entry of the block's table has to arrive where it belongs."""
    from mist_b200.config import load_config
    from mist_b200.inference import kv_cache
    from mist_b200.models.provider import base_model_provider
    from mist_b200.models.transformer import ParallelTransformer
    from mist_b200.ops import decode
    cfg, _ = load_config("config", ["experiment=gpt2-1.3b", f"model={model}", "model.num_hidden_layers=2",
                                    "model.hidden_size=512", "model.intermediate_size=1408",
                                    "model.num_attention_heads=8", "model.vocab_size=1024", "model.qkv_proj_bias=true",
                                    "model.out_proj_bias=true", "model.mlp_fc1_bias=true", "model.mlp_fc2_bias=true",
                                    "training.max_sequence_length=64", "strategy.layer_partitions=[2]"],
                         check_world_size=False)
    torch.manual_seed(b)
    net = base_model_provider(cfg.model, device=torch.device(DEV), dtype=torch.bfloat16).eval()
    stack = next(m for m in net.modules() if type(m) is ParallelTransformer)
    filled = 0
    with torch.no_grad():
        for name, p in stack.named_parameters():
            if p.dim() == 1:
                p.normal_(std=0.5).add_(1.0 if "norm" in name and name.endswith("weight") else 0.0)
                filled += 1
    assert filled >= 2 * (8 if model.startswith("gpt2") else 6)      # four biases and two norms a block
    x, res = (torch.randn(3, b, 1, 512, device=DEV, dtype=torch.bfloat16) for _ in range(2))

    def steps():
        with torch.no_grad(), kv_cache(net, b, 8) as ip:
            out = []
            for t in range(3):
                out.append(stack(x[t], res[t] if with_residual else None).float())
                ip.seqlen_offset += 1
            return torch.stack(out), [ip.key_value_memory[i][:, :3].float() for i in range(2)]

    calls = []
    native_step = decode.stack_step
    monkeypatch.setattr(decode, "stack_step", lambda *a: calls.append(native_step(*a)) or calls[-1])
    got, cache = steps()
    assert len(calls) == 3 and all(c is not None for c in calls)
    monkeypatch.setattr(decode, "stack_step", lambda *a: None)
    want, cache_ref = steps()
    # Two blocks of about ten roundings of at most 2^-9 each, at different places on the two sides: a 2-norm below
    # 2^-9 / sqrt(3) * sqrt(2 * 20), 0.7 %; a parameter in the wrong place changes half of the result and more.
    assert _rel(got, want) < 2 ** -6
    for a, r in zip(cache, cache_ref):
        assert _rel(a, r) < 2 ** -6
