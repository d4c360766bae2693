"""The framework's workloads at fixed sizes: training iterations of every model family, prompt
processing, single-token decoding, and attention over a long sequence.

Widths, head counts, vocabularies and sequence lengths are those of ``mist_b200/configs/model`` and of
the tests; a model is cut to a few of its layers, which leaves every kernel at its real size.  A case
is a dict of plain values; ``prepare`` makes what a program holds before the call, ``run`` is the call.
"""
import math

import torch

from mist_b200.api import build_training
from mist_b200.config import load_config
from mist_b200.inference import kv_cache
from mist_b200.models.provider import base_model_provider
from mist_b200.ops import functional as F

DEV = "cuda"
FAMILY = {"gpt": "gpt2/1.3b", "llama": "llama/1.3b", "falcon": "falcon/1.3b", "bert": "bert/1.3b", "t5": "t5/1.7b"}
GATED = ("llama",)


def listed():
    return [
        # the benchmark's layer (GPT-3 2.7B: 32 heads of 80) at its micro batch and sequence length: large GEMMs,
        # attention at an awkward head size, a full-size head and loss
        dict(name="train_gpt_2.7b_width", kind="train", family="gpt", hidden=2560, ffn=10240, heads=32, kv_heads=32,
             layers=4, batch=8, seq=2048, dec_seq=0, vocab=50304, micro_steps=1, ckpt=0),
        # the 7B preset: 4096 tokens, heads of 128, rotary, SwiGLU, two micro steps (fp32 gradient accumulation)
        # and one recomputed block; the largest case
        dict(name="train_llama_7b_width", kind="train", family="llama", hidden=4096, ffn=11008, heads=32, kv_heads=32,
             layers=2, batch=2, seq=4096, dec_seq=0, vocab=32000, micro_steps=2, ckpt=1),
        # parallel attention / MLP blocks with grouped-query heads at a middling width
        dict(name="train_falcon_gqa", kind="train", family="falcon", hidden=2048, ffn=8192, heads=16, kv_heads=4,
             layers=2, batch=4, seq=2048, dec_seq=0, vocab=50304, micro_steps=1, ckpt=0),
        # masked-LM training on right-padded batches of short sequences
        dict(name="train_bert_padded", kind="train", family="bert", hidden=2048, ffn=8192, heads=16, kv_heads=16,
             layers=4, batch=16, seq=512, dec_seq=0, vocab=50304, micro_steps=1, ckpt=0),
        # encoder-decoder: self and cross attention between sequences of different lengths
        dict(name="train_t5", kind="train", family="t5", hidden=2048, ffn=8192, heads=16, kv_heads=16,
             layers=2, batch=8, seq=512, dec_seq=128, vocab=50304, micro_steps=1, ckpt=0),
        # a small model on sequences that fill no tile: 7 x 1000 tokens
        dict(name="train_llama_350m_ragged", kind="train", family="llama", hidden=1024, ffn=2816, heads=16,
             kv_heads=16, layers=6, batch=7, seq=1000, dec_seq=0, vocab=50304, micro_steps=1, ckpt=0),
        # the smallest training step (tests, first runs): launches and host work decide
        dict(name="train_small", kind="train", family="gpt", hidden=512, ffn=2048, heads=4, kv_heads=4,
             layers=2, batch=2, seq=256, dec_seq=0, vocab=50304, micro_steps=1, ckpt=0),
        # prompt processing of two sequences into the key/value cache
        dict(name="prefill_llama_7b", kind="prefill", family="llama", hidden=4096, ffn=11008, heads=32, kv_heads=32,
             layers=4, batch=2, seq=1500, vocab=32000),
        # one token of one sequence: every weight is read for one row
        dict(name="decode_llama_7b_b1", kind="decode", family="llama", hidden=4096, ffn=11008, heads=32, kv_heads=32,
             layers=4, batch=1, seq=2047, vocab=32000),
        # one token of each of 32 sequences: the cache outweighs the weights
        dict(name="decode_gpt_2.7b_b32", kind="decode", family="gpt", hidden=2560, ffn=10240, heads=32, kv_heads=32,
             layers=4, batch=32, seq=1000, vocab=50304),
        # one token of a whole small model (24 layers): the latency of interactive generation
        dict(name="decode_llama_350m_b1", kind="decode", family="llama", hidden=1024, ffn=2816, heads=16, kv_heads=16,
             layers=24, batch=1, seq=120, vocab=50304),
        # attention alone over a long sequence, grouped-query heads, forward and backward
        dict(name="attention_long_gqa", kind="attention", heads=32, kv_heads=8, head_dim=128, batch=1, seq=16384,
             causal=True),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """One more case of the ranges above: any family, width, head size, sequence length and batch; at most
    three quarters of the largest listed case's operations."""
    most = 0.75 * max(work(c)["flops"] for c in listed())
    kind = rng.choice(["train", "train", "train", "prefill", "decode", "decode", "attention"])
    d = rng.choice([64, 80, 96, 128])
    if kind == "attention":
        kv = rng.choice([2, 4, 8])
        c = dict(kind=kind, heads=kv * rng.choice([1, 2, 4]), kv_heads=kv, head_dim=d, batch=rng.choice([1, 2, 3]),
                 seq=_log_int(rng, 200, 16384), causal=rng.random() < 0.8)
        while work(c)["flops"] > most / 4:
            c["seq"] = int(c["seq"] * 0.8)
        return c
    family = rng.choice(sorted(FAMILY)) if kind == "train" else rng.choice(["gpt", "llama"])
    heads = 4 * max(1, _log_int(rng, 512, 4096) // (4 * d))
    hidden = heads * d
    ffn = 4 * hidden if family not in GATED else (8 * hidden // 3 + 255) // 256 * 256
    kv = heads // 4 if family in ("falcon", "llama") and rng.random() < 0.3 else heads
    c = dict(kind=kind, family=family, hidden=hidden, ffn=ffn, heads=heads, kv_heads=kv, layers=rng.randint(1, 3),
             batch=1, seq=0, vocab=rng.choice([32000, 50304]))
    if kind == "decode":
        c["batch"] = _log_int(rng, 1, 48)
        c["seq"] = _log_int(rng, 16, 3000)
        return c
    c["seq"] = _log_int(rng, 100, 4096)
    tokens = _log_int(rng, max(1024, c["seq"]), 16384) if kind == "train" else _log_int(rng, c["seq"], 8192)
    c["batch"] = max(1, -(-tokens // c["seq"]) if kind == "train" else tokens // c["seq"])
    if kind == "train":
        c["dec_seq"] = max(16, c["seq"] // rng.choice([1, 3, 4])) if family == "t5" else 0
        c["micro_steps"] = rng.choice([1, 1, 2])
        c["ckpt"] = rng.choice([0, 0, 1])
    while work(c)["flops"] > most and (c["batch"] > 1 or c["layers"] > 1):
        c["batch"], c["layers"] = max(1, c["batch"] // 2), max(1, c["layers"] - 1)
    return c


# --------------------------------------------------------------------------------------- inputs
def _ids(shape, vocab, gen):
    """Token ids as the benchmark and the input providers draw them: uniform over the vocabulary.  (With the
    frequencies of text the rows of a few common tokens hold most of the embedding gradient's norm, and the
    rounding in them exceeds the root mean square of a table that is mostly zeros.)"""
    return torch.randint(0, vocab, shape, generator=gen, device=DEV)


def _overrides(c):
    n, g = c["layers"], c.get("micro_steps", 1)
    vec = [c["batch"], 1, 1, 0, 0, 0, 0, 0, 0, 0]
    seq = max(c["seq"], c.get("dec_seq", 0)) + (8 if c["kind"] in ("prefill", "decode") else 0)
    out = ["experiment=template-b200", f"model={FAMILY[c['family']]}", "hardware.num_gpus_per_node=1",
           f"model.hidden_size={c['hidden']}", f"model.intermediate_size={c['ffn']}",
           f"model.num_attention_heads={c['heads']}", f"model.num_heads_kv={c['kv_heads']}",
           f"model.num_hidden_layers={n}", f"model.vocab_size={c['vocab']}", f"training.vocab_size={c['vocab']}",
           f"training.max_sequence_length={seq}", f"training.global_batch_size={c['batch'] * g}",
           f"strategy.layer_partitions=[{n}]", "strategy.device_assignment=[[1,1]]",
           f"strategy.gradient_checkpointing=[{min(c.get('ckpt', 0), n)}]",
           f"strategy.gradient_accumulation_steps={g}", f"strategy.stage_strategies=[{vec}]".replace(" ", ""),
           f"strategy.pre_post_strategy_array={vec}".replace(" ", "")]
    if c["family"] == "llama":
        out.append("model.rotary_emb_fraction=1.0")
    return out


def _train_batch(c, gen):
    rows, s, v = c["batch"] * c["micro_steps"], c["seq"], c["vocab"]
    ids = _ids((rows, s + 1), v, gen)
    inp, nxt = ids[:, :-1].contiguous(), ids[:, 1:].contiguous()
    if c["family"] == "bert":
        # lengths between a quarter and all of the positions, 15 % of the real tokens are predicted
        lens = (s * (0.25 + 0.75 * torch.rand(rows, generator=gen, device=DEV))).long().clamp_(1, s)
        mask = torch.arange(s, device=DEV)[None] < lens[:, None]
        chosen = (torch.rand(rows, s, generator=gen, device=DEV) < 0.15) & mask
        return {"input_ids": inp, "attention_mask": mask.long(),
                "lm_labels": torch.where(chosen, nxt, torch.full_like(nxt, -100))}
    if c["family"] == "t5":
        dec = _ids((rows, c["dec_seq"] + 1), v, gen)
        return {"encoder_input_ids": inp, "decoder_input_ids": dec[:, :-1].contiguous(),
                "lm_labels": dec[:, 1:].contiguous()}
    return {"input_ids": inp, "labels": nxt}


def prepare(case, seed):
    c = case
    gen = torch.Generator(device=DEV).manual_seed(seed)
    if c["kind"] == "attention":
        def rand(heads):
            return torch.randn(c["batch"], c["seq"], heads, c["head_dim"], generator=gen, device=DEV,
                               dtype=torch.bfloat16)
        q, k, v = (rand(n).requires_grad_(True) for n in (c["heads"], c["kv_heads"], c["kv_heads"]))
        return dict(case=c, q=q, k=k, v=v, dout=rand(c["heads"]))
    if c["kind"] == "train":
        session = build_training("config", _overrides(c), seed=seed)
        return dict(case=c, session=session, batch=_train_batch(c, gen))
    cfg, _ = load_config("config", _overrides(c))
    torch.manual_seed(seed)
    model = base_model_provider(cfg.model, device=torch.device(DEV), dtype=torch.bfloat16).eval()
    b, s = c["batch"], c["seq"]
    ids = _ids((b, s + 1), c["vocab"], gen)
    holder = kv_cache(model, b, s + 8)
    ip = holder.__enter__()
    state = dict(case=c, model=model, holder=holder, ip=ip, prompt=ids[:, :s].contiguous(),
                 token=ids[:, s:].contiguous())
    if c["kind"] == "decode":
        with torch.no_grad():
            _forward(state, state["prompt"])
    return state


# ------------------------------------------------------------------------------------------ pass
def _forward(state, ids):
    """One call of the generation loop: positions from the cache's fill, logits, the fill moved on."""
    ip, b, n = state["ip"], ids.shape[0], ids.shape[1]
    pos = torch.arange(ip.seqlen_offset, ip.seqlen_offset + n, device=ids.device)
    logits = state["model"](ids, position_ids=pos.unsqueeze(0).expand(b, -1))
    ip.seqlen_offset += n
    return logits


def run(state):
    c = state["case"]
    if c["kind"] == "attention":
        q, k, v = state["q"], state["k"], state["v"]
        o = F.attention(q, k, v, causal=c["causal"])
        return (o,) + torch.autograd.grad(o, (q, k, v), state["dout"])
    if c["kind"] == "train":
        session = state["session"]
        if c["family"] in ("bert", "t5"):
            loss = session.step_on_device_batch(state["batch"])
        else:
            loss = session.step_on_device(state["batch"]["input_ids"], state["batch"]["labels"])
        session.engine.finish()
        units = session.engine.units
        return dict(loss=loss, grads=[u.flat_grad for u in units], weights=[u.master for u in units])
    ip = state["ip"]
    with torch.no_grad():
        if c["kind"] == "prefill":
            ip.reset()
            logits = _forward(state, state["prompt"])
        else:
            ip.seqlen_offset = c["seq"]
            logits = _forward(state, state["token"])
    return dict(logits=logits, cache=[ip.key_value_memory[i] for i in sorted(ip.key_value_memory)])


# ------------------------------------------------------------------------------------------ work
def work(case):
    """Operations: the products of the weights with the tokens (three times for a training step, once more
    for a recomputed block) and of attention over the visible positions.  Bytes: each weight, optimizer
    value, gradient, cache entry, input and result once."""
    c = case
    if c["kind"] == "attention":
        b, s, d = c["batch"], c["seq"], c["head_dim"]
        pairs = b * c["heads"] * s * (s + 1) / 2 if c["causal"] else b * c["heads"] * s * s
        q, kv = b * s * c["heads"] * d * 2, b * s * c["kv_heads"] * d * 2
        # forward: two products per pair; backward: five
        return {"flops": 7 * 2 * d * pairs, "bytes": 4 * q + 4 * kv}       # q, dout, o, dq; k, v, dk, dv
    h, f, n, v = c["hidden"], c["ffn"], c["layers"], c["vocab"]
    kvh = h // c["heads"] * c["kv_heads"]
    mlp = (3 if c["family"] in GATED else 2) * h * f
    attn = 2 * h * h + 2 * h * kvh
    b, s = c["batch"], c["seq"]
    if c["kind"] != "train":
        new = s if c["kind"] == "prefill" else 1
        pairs = b * s * (s + 1) / 2 if c["kind"] == "prefill" else b * (s + 1)
        flops = 2 * b * new * (n * (attn + mlp) + v * h) + 4 * h * n * pairs
        cache = n * 2 * kvh * 2 * b * (new + (s if c["kind"] == "decode" else 0))
        return {"flops": flops, "bytes": 2 * (n * (attn + mlp) + v * h + b * new * h) + cache + 2 * b * new * v}
    g = c["micro_steps"]
    ckpt = min(c["ckpt"], n)
    if c["family"] == "t5":
        dt, td = b * c["dec_seq"], c["dec_seq"]
        fwd_enc = 2 * b * s * (attn + mlp) + 4 * h * b * s * s
        fwd_dec = (2 * dt * (attn + 2 * h * h + mlp) + 2 * b * s * 2 * h * h
                   + 4 * h * b * (td * (td + 1) / 2 + td * s))
        block, params, tokens = fwd_enc + fwd_dec, n * (3 * attn + 2 * mlp) + v * h, dt
    else:
        pairs = b * s * s if c["family"] == "bert" else b * s * (s + 1) / 2
        block, tokens = 2 * b * s * (attn + mlp) + 4 * h * pairs, b * s
        params = n * (attn + mlp) + v * h * (1 if c["family"] == "bert" else 2)
    flops = g * (block * (3 * n + ckpt) + 6 * tokens * h * v)
    # weights read and written, gradients written, master weights and two moments read and written
    return {"flops": flops, "bytes": params * (2 + 2 + (4 if g > 1 else 2) + 24) + 16 * g * b * (s + c["dec_seq"])}


def tolerance(case):
    """Measured: the same pass with the library GEMMs and attention in place of the framework's, both in bf16.
    Training: gradients of the listed cases and of drawn ones differ by 0.002 to 0.014 (2-norm), single values of
    the sparse embedding gradients by up to 0.5 of its root mean square.  Inference: 0.008, 0.04.  Attention: 0.0018,
    0.13 (first rows of a causal mask, few terms)."""
    if case["kind"] == "train":
        return {"rel": 0.03, "max": 0.99}
    if case["kind"] == "attention":
        return {"rel": 0.008, "max": 0.5}
    return {"rel": 0.03, "max": 0.2}
