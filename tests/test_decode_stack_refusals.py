"""The native decoding step takes only stacks whose modules would do exactly what it does."""
import pytest
import torch
from torch.nn.modules import module as nn_module

from mist_b200.config import load_config
from mist_b200.inference import kv_cache
from mist_b200.models.provider import base_model_provider
from mist_b200.models.transformer import ParallelTransformerLayer
from mist_b200.ops import decode

BF16 = torch.bfloat16


def _model(device, kind="gpt2/1.3b"):
    cfg, _ = load_config("config", ["experiment=gpt2-1.3b", f"model={kind}", "model.num_hidden_layers=2",
                                    "model.hidden_size=64", "model.intermediate_size=128", "model.vocab_size=128",
                                    "model.num_attention_heads=4", "training.max_sequence_length=16",
                                    "strategy.layer_partitions=[2]"], check_world_size=False)
    torch.manual_seed(0)
    net = base_model_provider(cfg.model, device=torch.device(device), dtype=BF16).eval()
    return net, [m for m in net.modules() if type(m) is ParallelTransformerLayer]


def _plain_attribute(mod, name, value):
    del mod._parameters[name]
    object.__setattr__(mod, name, value)


def _weight(mod, value):
    mod.weight = torch.nn.Parameter(value)


def _unaligned(shape):
    n = torch.Size(shape).numel()
    return torch.zeros(n + 8, dtype=BF16)[4:4 + n].view(shape)


# each change to the second block or to the call, and the general path has to take over
CHANGES = {
    "forward_of_an_instance": lambda c: setattr(c.layer.attn.out_proj, "forward", lambda x, residual=None: x),
    "forward_of_the_norm": lambda c: setattr(c.layer.norm2, "forward", c.layer.norm2.forward),
    "forward_of_the_block": lambda c: setattr(c.layer, "forward", c.layer.forward),
    "hook": lambda c: c.layer.mlp.fc2.register_forward_hook(lambda *a: None),
    "pre_hook": lambda c: c.layer.attn.register_forward_pre_hook(lambda *a: None),
    "global_hook": lambda c: nn_module.register_module_forward_hook(lambda *a: None),
    "global_pre_hook": lambda c: nn_module.register_module_forward_pre_hook(lambda *a: None),
    "computed_weight": lambda c: _plain_attribute(c.layer.mlp.fc1, "weight", c.layer.mlp.fc1.weight.detach()),
    "computed_bias": lambda c: _plain_attribute(c.layer.norm1, "bias", torch.ones(64, dtype=BF16)),
    "bias_set_later": lambda c: object.__setattr__(c.layer.attn.Wqkv, "bias", torch.ones(192, dtype=BF16)),
    "fp32_weight": lambda c: _weight(c.layer.mlp.fc1, torch.zeros(128, 64)),
    "narrow_weight": lambda c: _weight(c.layer.attn.Wqkv, torch.zeros(192, 32, dtype=BF16)),
    "short_weight": lambda c: _weight(c.layer.attn.Wqkv, torch.zeros(128, 64, dtype=BF16)),
    "transposed_weight": lambda c: _weight(c.layer.mlp.fc2, torch.zeros(128, 64, dtype=BF16)),
    "strided_weight": lambda c: _weight(c.layer.attn.out_proj, torch.zeros(64, 64, dtype=BF16).t()),
    "unaligned_weight": lambda c: _weight(c.layer.attn.out_proj, _unaligned((64, 64))),
    "short_norm": lambda c: _weight(c.layer.norm2, torch.ones(32, dtype=BF16)),
    "weight_without_storage": lambda c: _weight(c.layer.mlp.fc2, torch.zeros(64, 128, dtype=BF16, device="meta")),
    "dropout": lambda c: (setattr(c.layer, "hidden_dropout", 0.1), c.layer.train()),
    "wide_hidden": lambda c: setattr(c, "hidden", torch.zeros(2, 1, 128, dtype=BF16)),
    "two_tokens": lambda c: setattr(c, "hidden", torch.zeros(2, 2, 64, dtype=BF16)),
    "fp32_residual": lambda c: setattr(c, "residual", torch.zeros(2, 1, 64)),
    "short_residual": lambda c: setattr(c, "residual", torch.zeros(1, 1, 64, dtype=BF16)),
    "full_cache": lambda c: setattr(c.ip, "seqlen_offset", 8),
    "short_cache": lambda c: c.ip.key_value_memory.update({1: torch.zeros(3, 4, 2, 4, 16, dtype=BF16)}),
    "small_cache": lambda c: c.ip.key_value_memory.update({1: torch.zeros(1, 8, 2, 4, 16, dtype=BF16)}),
}


class _Call:
    pass


@pytest.mark.parametrize("change", [None, *CHANGES])
def test_refusals(change):
    net, layers = _model("cpu")
    c = _Call()
    c.layer, c.hidden, c.residual = layers[1], torch.zeros(2, 1, 64, dtype=BF16), None
    with torch.no_grad(), kv_cache(net, 3, 8) as c.ip:
        c.ip.seqlen_offset = 5
        assert decode._stack(layers, c.hidden, c.residual) is not None
        assert decode._block(c.layer, 64, 0, []) is None          # its weights are not on that device
        made = CHANGES[change](c) if change else None
        try:
            assert (decode._stack(layers, c.hidden, c.residual) is None) == (change is not None)
        finally:
            if change and change.startswith("global"):
                made.remove()


def test_batch_limit():
    net, layers = _model("cpu", "llama/1.3b")
    with torch.no_grad(), kv_cache(net, 129, 2):
        assert decode._stack(layers, torch.zeros(128, 1, 64, dtype=BF16), None) is not None
        assert decode._stack(layers, torch.zeros(129, 1, 64, dtype=BF16), None) is None


@pytest.mark.parametrize("name,value", [("gemm_backend", "cublas"), ("gemm_max_ctas", 100)])
def test_settings(name, value, monkeypatch):
    net, layers = _model("cpu")
    monkeypatch.setattr(decode.Settings, name, value)
    with torch.no_grad(), kv_cache(net, 1, 2):
        assert decode._stack(layers, torch.zeros(1, 1, 64, dtype=BF16), None) is None


@pytest.mark.gpu
@pytest.mark.parametrize("change", ["forward", "global_hook"])
def test_replaced_forwards_run(change):
    net, layers = _model("cuda")
    seen = []
    if change == "forward":
        own = layers[1].attn.out_proj.forward
        layers[1].attn.out_proj.forward = lambda x, residual=None: seen.append(1) or own(x, residual=residual)
        handle = None
    else:
        handle = nn_module.register_module_forward_hook(lambda mod, *a: seen.append(mod))
    try:
        with torch.no_grad(), kv_cache(net, 2, 8):
            net(torch.zeros(2, 1, dtype=torch.long, device="cuda"), position_ids=torch.zeros(2, 1, dtype=torch.long,
                                                                                             device="cuda"))
    finally:
        if handle is not None:
            handle.remove()
    assert seen and (change == "forward" or layers[1].attn.out_proj in seen)
