"""What the streamed decode step is handed is checked on the host before a kernel gets its address.

The library is replaced by a recorder, so nothing runs: a call with tensors that do not fit must not reach the kernel
that would read or write past them (the caches of ``rope_append``, the operands of the projections)."""

import types

import pytest
import torch

from interattn_b200 import llama_step

BF = torch.bfloat16
B, HQ, HKV, D, HIDDEN, INTER, VOCAB, T = 3, 4, 2, 64, 256, 512, 320, 48


class _Library:
    """Takes any call and remembers its name; sizes are answered with a constant."""

    def __init__(self):
        self.calls = []

    def __getattr__(self, name):
        def call(*args):
            self.calls.append(name)
            return 1 << 20 if name.endswith("_bytes") else 0
        return call


class _Attention:
    """Stands for the layer's ``DecodeAttention``."""

    def __init__(self, out):
        self.out = out

    def step(self, q):
        return self.out


def _step(monkeypatch):
    lib = _Library()
    monkeypatch.setattr(llama_step._lib, "load", lambda: lib)
    monkeypatch.setattr(llama_step, "_stream", lambda: None)
    monkeypatch.setattr(llama_step, "_need_cuda", lambda *a: None)
    linear = lambda n, k: types.SimpleNamespace(weight=torch.zeros(n, k, dtype=BF))  # noqa: E731
    norm = lambda: types.SimpleNamespace(weight=torch.ones(HIDDEN, dtype=BF))  # noqa: E731
    layer = types.SimpleNamespace(
        self_attn=types.SimpleNamespace(q_proj=linear(HQ * D, HIDDEN), k_proj=linear(HKV * D, HIDDEN),
                                        v_proj=linear(HKV * D, HIDDEN), o_proj=linear(HIDDEN, HQ * D)),
        mlp=types.SimpleNamespace(gate_proj=linear(INTER, HIDDEN), up_proj=linear(INTER, HIDDEN),
                                  down_proj=linear(HIDDEN, INTER)),
        input_layernorm=norm(), post_attention_layernorm=norm())
    rotary = lambda x, pos: (torch.zeros(1, pos.shape[1], D, dtype=BF),) * 2  # noqa: E731
    core = types.SimpleNamespace(embed_tokens=linear(VOCAB, HIDDEN), layers=[layer], norm=norm(), rotary_emb=rotary)
    model = types.SimpleNamespace(model=core, lm_head=linear(VOCAB, HIDDEN), config=types.SimpleNamespace(
        rms_norm_eps=1e-5, num_attention_heads=HQ, num_key_value_heads=HKV, head_dim=D, hidden_size=HIDDEN,
        intermediate_size=INTER))
    cache = types.SimpleNamespace(layers=[types.SimpleNamespace(keys=torch.zeros(B, HKV, T, D, dtype=BF),
                                                                values=torch.zeros(B, HKV, T, D, dtype=BF))])
    step = llama_step.FusedLlamaStep(model, cache, [_Attention(torch.zeros(B, HQ, D, dtype=BF))],
                                     torch.ones(B, dtype=torch.int32), T)
    step.parts = torch.empty(1 << 20, dtype=torch.uint8)   # the streamed form, on tensors of this machine
    return step, lib


def _zeros(*shape, dtype=BF):
    return torch.zeros(shape, dtype=dtype)


def test_fitting_tensors_take_the_streamed_form(monkeypatch):
    step, lib = _step(monkeypatch)
    step._stream_step(_zeros(B, 1, dtype=torch.int64))
    assert lib.calls.count("ia_llama_gemm_parts") == 5 and lib.calls[-1] == "ia_llama_argmax_parts"


# refused: the other form, which such a step is left to, raises the ValueError of rope_append; the rest it can judge
# for itself (torch.mm)
@pytest.mark.parametrize("change,refused", [
    (dict(k=_zeros(B - 1, HKV, T, D), v=_zeros(B - 1, HKV, T, D)), True),      # a cache for fewer sequences
    (dict(k=_zeros(B, HKV - 1, T, D), v=_zeros(B, HKV - 1, T, D)), True),      # fewer kv heads
    (dict(k=_zeros(B, HKV, T, D // 2), v=_zeros(B, HKV, T, D // 2)), True),    # smaller heads
    (dict(v=_zeros(B, HKV, T - 16, D)), True),                                 # V shorter than K
    (dict(k=_zeros(B, HKV, T, D, dtype=torch.float32)), True),
    (dict(k=_zeros(B, T, HKV, D).transpose(1, 2)), True),                      # the same shape, other strides
    (dict(seq_lens=torch.ones(B, dtype=torch.int64)), True),
    (dict(seq_lens=torch.ones(B - 1, dtype=torch.int32)), True),
    (dict(seq_lens=torch.ones(2 * B, dtype=torch.int32)[::2]), False),
    (dict(w_qkv=_zeros((HQ + 2 * HKV) * D - 8, HIDDEN)), False),               # fewer columns than the consumer reads
], ids=["batch", "kv_heads", "head_dim", "v_shorter", "dtype", "strides", "int64_lens", "short_lens", "strided_lens",
        "w_qkv"])
def test_the_cache_append_is_not_reached(change, refused, monkeypatch):
    step, lib = _step(monkeypatch)
    for name, t in change.items():
        if name == "seq_lens":
            step.seq_lens = t
        else:
            step.layers[0][name] = t
    tokens = _zeros(B, 1, dtype=torch.int64)
    step._stream_step(tokens)
    assert not [c for c in lib.calls if c.endswith("_parts")], lib.calls
    if refused:
        with pytest.raises(ValueError):
            step.step(tokens)
        assert "ia_llama_rope_append" not in lib.calls


@pytest.mark.parametrize("name,weight", [("w_o", _zeros(HIDDEN, HQ * D + 8)), ("w_gu", _zeros(2 * INTER - 16, HIDDEN)),
                                         ("w_down", _zeros(HIDDEN, INTER).t()), ("norm2", _zeros(HIDDEN - 8)),
                                         ("w_o", _zeros(HIDDEN, HQ * D + 1)[:, 1:]), ("lm_head", _zeros(VOCAB + 8, HIDDEN)),
                                         ("context", _zeros(B, HQ, D, dtype=torch.float32)),
                                         ("context", _zeros(1 + B * HQ * D)[1:].view(B, HQ, D))],
                         ids=["w_o", "w_gu", "w_down", "norm2", "w_o_strided", "lm_head", "context_f32", "context_odd"])
def test_no_projection_reads_an_operand_that_does_not_fit(name, weight, monkeypatch):
    """Weights exchanged after the construction, an attention output of another type or off its alignment."""
    step, lib = _step(monkeypatch)
    if name == "context":
        step.attention[0].out = weight
    elif name == "lm_head":
        step.lm_head = weight
    else:
        step.layers[0][name] = weight
    step._stream_step(_zeros(B, 1, dtype=torch.int64))
    assert lib.calls.count("ia_llama_gemm_parts") == (1 if name == "context" else 0), lib.calls
    assert "ia_llama_argmax_parts" not in lib.calls
