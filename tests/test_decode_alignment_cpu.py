"""Tensors that do not start on 16 bytes never reach the decode kernels, whose loads take 16 bytes at a time."""
import ctypes

import pytest
import torch

from mist_b200.ops import functional as F
from mist_b200.ops import native


def _at(offset, *shape):
    """A contiguous bf16 tensor that starts ``offset`` elements behind a 16-byte boundary."""
    n = torch.Size(shape).numel()
    flat = torch.randn(n + 16).to(torch.bfloat16)
    start = (-flat.data_ptr() % 16) // 2 + offset
    return flat[start:start + n].view(shape)


# elements in front of q, k and v: strides are multiples of 8 throughout, only the start is off
@pytest.mark.parametrize("q_off,k_off,v_off", [(0, 0, 0), (4, 0, 0), (1, 0, 0), (0, 4, 0), (0, 0, 2), (4, 4, 4)])
def test_decode_attention_pointers(q_off, k_off, v_off, monkeypatch):
    b, nh, d, rows = 2, 3, 16, 6
    q = _at(q_off, b, 8 * nh * d)[:, :nh * d].view(b, nh, d)
    k, v = _at(k_off, b, rows, nh, d), _at(v_off, b, rows, nh, d)
    want = F.decode_attention(q, k, v, 5)              # on the CPU: in torch
    launched = []

    def call(name, q_at, k_at, v_at, out_at, *rest):
        launched.append(name)
        assert (q_at | k_at | v_at) % 16 == 0 and not any(s % 8 for s in rest[5:12])
        got = (ctypes.c_uint16 * (b * nh * d)).from_address(q_at)
        if q_off:                                      # a copy of q, and the right one
            assert torch.frombuffer(bytearray(got), dtype=torch.bfloat16).equal(q.reshape(-1))
    monkeypatch.setattr(F, "use_native", lambda *t: True)
    monkeypatch.setattr(F, "stream", lambda: 0)
    monkeypatch.setattr(F, "call", call)
    out = F.decode_attention(q, k, v, 5)
    assert bool(launched) == (k_off == v_off == 0)
    if not launched:
        torch.testing.assert_close(out, want)


@pytest.mark.parametrize("qkv_off,cache_off", [(0, 0), (4, 0), (0, 4)])
def test_rope_append_pointers(qkv_off, cache_off, monkeypatch):
    monkeypatch.setattr(F, "use_native", lambda *t: True)
    qkv, cache = _at(qkv_off, 1, 1, 48), _at(cache_off, 1, 4, 2, 1, 16)
    assert F.rope_append_available(qkv, cache, 0, 16) == (qkv_off == cache_off == 0)


def test_entry_points_refuse_them():
    if not native.kernels_path().exists():
        pytest.skip("the kernels library is not built")
    lib = ctypes.CDLL(str(native.kernels_path()))
    p, i, n = ctypes.c_void_p, ctypes.c_int, ctypes.c_long
    lib.mb_decode_attn.argtypes = [p] * 4 + [i] * 5 + [n] * 7 + [ctypes.c_float, i, p]
    lib.mb_rope_append.argtypes = [p] * 4 + [i] * 7 + [n, i, p]
    for bad in range(3):               # refused before anything is launched
        at = [4096 + (8 if j == bad else 0) for j in range(3)]
        assert lib.mb_decode_attn(*at, 4096, 1, 1, 1, 16, 4, *[16] * 7, 1.0, 0, 0) == -1
    for at in ((4104, 4096), (4096, 4104)):
        assert lib.mb_rope_append(*at, 0, 0, 1, 1, 1, 1, 16, 0, 0, 64, 0, 0) == -1
