"""One batched Llama decode step with every non-GEMM op a single fused launch.

The reference decodes through the unmodified Hugging Face model and replaces
only ``eager_attention_forward`` (``condition_block_triton_impl/core.py:1372-1379``);
its captured step (``core.py:190-316``) therefore replays the model's own
element-wise PyTorch kernels - about forty per layer - around the attention hook.
``FusedLlamaStep`` runs the same arithmetic, on the same weights and the same
static cache, as ten launches per layer:

    add+RMSNorm | QKV GEMM | RoPE+cache append | block selection | sparse attention
    | O GEMM | add+RMSNorm | gate/up GEMM | SiLU*up | down GEMM

For batches of at most 16 rows the GEMMs run on ``csrc/skinny_gemm.cu`` (a tcgen05 kernel that streams the
weights as the model holds them and leaves partial sums to the element-wise kernel that follows); larger batches
and ``own_gemm="none"`` use ``torch.mm`` (cuBLAS) on the same concatenated weights.  Everything else is ``csrc/llama_step.cu`` and the attention kernels, keeping the
bf16 rounding points of ``transformers.models.llama.modeling_llama`` so that the
fused and the module-by-module step agree up to fp32 summation order.
"""

from __future__ import annotations

from typing import Optional

import torch

from . import _lib
from .ops import _need_cuda, _ptr, _stream


def _bf16(*tensors):
    for t in tensors:
        if t is not None and (t.dtype != torch.bfloat16 or not t.is_contiguous()):
            raise ValueError("contiguous bfloat16 tensors are needed")


def add_rmsnorm(residual: torch.Tensor, delta: Optional[torch.Tensor], weight: torch.Tensor, eps: float,
                out: torch.Tensor) -> torch.Tensor:
    """``residual += delta`` (skipped for ``None``), then ``out = weight * rmsnorm(residual)``; rows [n, hidden]."""
    _need_cuda(residual)
    _bf16(residual, delta, weight, out)
    n, hidden = residual.shape
    if out.shape != residual.shape or (delta is not None and delta.shape != residual.shape) or weight.numel() != hidden:
        raise ValueError("add_rmsnorm: shapes differ")
    _lib.check(_lib.load().ia_llama_add_rmsnorm(_ptr(residual), _ptr(delta) if delta is not None else None,
                                                _ptr(weight), _ptr(out), n, hidden, float(eps), _stream()))
    return out


def rope_append(qkv: torch.Tensor, cos: torch.Tensor, sin: torch.Tensor, seq_lens: torch.Tensor,
                k_cache: torch.Tensor, v_cache: torch.Tensor, q_out: torch.Tensor) -> torch.Tensor:
    """Rotate the q and k heads of ``qkv [B, (Hq + 2 Hkv) * D]`` at position ``seq_lens - 1``, write k and v
    into the static cache tensors ``[B, Hkv, T, D]`` there and q into ``q_out [B, Hq, D]``."""
    _need_cuda(qkv)
    _bf16(qkv, cos, sin, k_cache, v_cache, q_out)
    b, hkv, t, d = (int(x) for x in k_cache.shape)
    hq = int(q_out.shape[1])
    if qkv.shape != (b, (hq + 2 * hkv) * d) or q_out.shape != (b, hq, d) or v_cache.shape != k_cache.shape:
        raise ValueError("rope_append: shapes differ")
    if cos.shape != sin.shape or cos.dim() != 2 or cos.shape[1] != d:
        raise ValueError("rope_append: cos/sin are [positions, head_dim]")
    if seq_lens.dtype != torch.int32 or seq_lens.numel() != b:
        raise ValueError("rope_append: seq_lens is int32 [batch]")
    _lib.check(_lib.load().ia_llama_rope_append(
        _ptr(qkv), _ptr(cos), _ptr(sin), int(cos.shape[0]), _ptr(seq_lens), _ptr(k_cache), _ptr(v_cache),
        hkv * t * d, t * d, t, _ptr(q_out), b, hq, hkv, d, _stream()))
    return q_out


def silu_mul(gate_up: torch.Tensor, out: torch.Tensor) -> torch.Tensor:
    """``out = silu(gate_up[:, :I]) * gate_up[:, I:]``."""
    _need_cuda(gate_up)
    _bf16(gate_up, out)
    n, two_i = gate_up.shape
    if two_i % 2 or out.shape != (n, two_i // 2):
        raise ValueError("silu_mul: shapes differ")
    _lib.check(_lib.load().ia_llama_silu_mul(_ptr(gate_up), _ptr(out), n, two_i // 2, _stream()))
    return out


def argmax(logits: torch.Tensor, out: torch.Tensor) -> torch.Tensor:
    """Row-wise arg-max of bf16 ``logits [n, vocab]`` into int64 ``out`` (n elements); lowest index on ties."""
    _need_cuda(logits)
    if logits.dtype != torch.bfloat16 or logits.dim() != 2 or logits.stride(1) != 1:
        raise ValueError("argmax: bfloat16 [rows, vocab] with unit inner stride")
    if out.dtype != torch.int64 or out.numel() != logits.shape[0] or not out.is_contiguous():
        raise ValueError("argmax: out is a contiguous int64 tensor with one element per row")
    _lib.check(_lib.load().ia_llama_argmax(_ptr(logits), int(logits.stride(0)), int(logits.shape[0]),
                                           int(logits.shape[1]), _ptr(out), _stream()))
    return out


def gemm_workspace(n: int, device) -> torch.Tensor:
    """Zeroed scratch for ``gemm`` calls with at most ``n`` output columns (one per stream)."""
    size = int(_lib.load().ia_llama_gemm_workspace_bytes(int(n)))
    return torch.zeros(size, dtype=torch.uint8, device=device)


class PackedWeight:
    """A linear layer's weight ``[n, k]`` in the tile order ``gemm`` streams it (packed once)."""

    def __init__(self, w: torch.Tensor):
        _need_cuda(w)
        _bf16(w)
        if w.dim() != 2:
            raise ValueError("a [n, k] weight is needed")
        self.n, self.k = int(w.shape[0]), int(w.shape[1])
        lib = _lib.load()
        self.data = torch.empty(int(lib.ia_llama_gemm_packed_bytes(self.n, self.k)), dtype=torch.uint8,
                                device=w.device)
        _lib.check(lib.ia_llama_gemm_pack(_ptr(w), self.n, self.k, _ptr(self.data), _stream()))


def gemm(x: torch.Tensor, w: PackedWeight, out: torch.Tensor, workspace: torch.Tensor) -> torch.Tensor:
    """``out [m, n] = x [m, k] @ w [n, k].T`` for m <= 32 (``nn.Linear`` without bias)."""
    _need_cuda(x)
    _bf16(x, out)
    m, k = x.shape
    if k != w.k or out.shape != (m, w.n):
        raise ValueError("gemm: shapes differ")
    _lib.check(_lib.load().ia_llama_gemm(_ptr(x), _ptr(w.data), _ptr(out), m, w.n, k, _ptr(workspace),
                                         int(workspace.numel()), _stream()))
    return out


class FusedLlamaStep:
    """Decode step of a Hugging Face ``LlamaForCausalLM`` over its ``StaticCache``.

    ``attention[i]`` is the ``ops.DecodeAttention`` of layer ``i`` (its ``PagedKV`` views the
    cache tensors in place and shares ``seq_lens``).  ``step(tokens)`` consumes ``tokens
    [B, 1]`` int64, writes the next greedy tokens into it and leaves the logits in
    ``self.logits``.  The position of the incoming token is ``seq_lens - 1`` for every
    sequence; the caller advances ``seq_lens`` between steps.  Nothing is allocated inside
    ``step``: it can be captured into a CUDA graph."""

    PROJECTIONS = ("w_qkv", "w_o", "w_gu", "w_down", "lm_head")

    def __init__(self, model, cache, attention, seq_lens: torch.Tensor, cache_len: int,
                 own_gemm: Optional[str] = None):
        # own_gemm: None reads INTERATTN_B200_LLAMA_GEMM; when that is unset too, batches of at most 16 rows
        # stream all projections (see _stream_step).  A name pins the form: "none" = torch.mm (cuBLAS), "all" or a
        # comma-separated subset of PROJECTIONS = those on the packed-weight kernel, the others on torch.mm.
        # Batches above 32 rows always use torch.mm.
        import os
        if own_gemm is None:
            own_gemm = os.environ.get("INTERATTN_B200_LLAMA_GEMM")
        streaming = own_gemm is None
        if streaming:
            own_gemm = "none"
        if own_gemm == "all":
            own = set(self.PROJECTIONS)
        elif own_gemm in ("none", "cublas", ""):
            own = set()
        else:
            own = {name.strip() for name in own_gemm.split(",")}
            if not own <= set(self.PROJECTIONS):
                raise ValueError(f"own_gemm names must come from {self.PROJECTIONS}")
        cfg = model.config
        if getattr(cfg, "attention_bias", False) or getattr(cfg, "mlp_bias", False):
            raise ValueError("projection biases are not supported")
        core = model.model
        p0 = core.embed_tokens.weight
        if p0.dtype != torch.bfloat16:
            raise ValueError("a bfloat16 model is needed")
        self.embed = p0
        self.eps = float(cfg.rms_norm_eps)
        self.seq_lens = seq_lens
        self.attention = list(attention)
        self.hq, self.hkv = int(cfg.num_attention_heads), int(cfg.num_key_value_heads)
        self.d = int(getattr(cfg, "head_dim", None) or cfg.hidden_size // cfg.num_attention_heads)
        self.layers = []
        for i, layer in enumerate(core.layers):
            a, m = layer.self_attn, layer.mlp
            self.layers.append(dict(
                norm1=layer.input_layernorm.weight, norm2=layer.post_attention_layernorm.weight,
                w_qkv=torch.cat([a.q_proj.weight, a.k_proj.weight, a.v_proj.weight], dim=0).contiguous(),
                w_o=a.o_proj.weight, w_gu=torch.cat([m.gate_proj.weight, m.up_proj.weight], dim=0).contiguous(),
                w_down=m.down_proj.weight, k=cache.layers[i].keys, v=cache.layers[i].values))
        self.final_norm = core.norm.weight
        self.lm_head = model.lm_head.weight
        b = int(seq_lens.numel())
        dev, h, inter = p0.device, int(cfg.hidden_size), int(cfg.intermediate_size)
        q_cols, kv_cols = self.hq * self.d, self.hkv * self.d
        self._layer_shapes = (("norm1", (h,)), ("w_qkv", (q_cols + 2 * kv_cols, h)), ("w_o", (h, q_cols)),
                              ("norm2", (h,)), ("w_gu", (2 * inter, h)), ("w_down", (h, inter)))
        with torch.no_grad():
            pos = torch.arange(cache_len, device=dev)[None, :]
            cos, sin = core.rotary_emb(torch.empty((1,), dtype=torch.bfloat16, device=dev), pos)
        self.cos, self.sin = cos[0].contiguous(), sin[0].contiguous()
        new = lambda *shape: torch.empty(shape, dtype=torch.bfloat16, device=dev)  # noqa: E731
        # the streamed form writes neither o, down, qkv nor gu; they are there for a step that has to leave it
        self.x, self.h, self.o, self.down = new(b, h), new(b, h), new(b, h), new(b, h)
        self.qkv, self.q = new(b, (self.hq + 2 * self.hkv) * self.d), new(b, self.hq, self.d)
        self.gu, self.act = new(b, 2 * inter), new(b, inter)
        self.logits = new(b, int(self.lm_head.shape[0]))
        self.own_gemm = set() if b > 32 else own
        self.gemm_ws = None
        if self.own_gemm:   # pack the chosen projections once (their concatenated copies are then dropped)
            self.gemm_ws = gemm_workspace(int(self.lm_head.shape[0]), dev)
            for L in self.layers:
                for name in self.own_gemm - {"lm_head"}:
                    L[name] = PackedWeight(L[name])
            if "lm_head" in self.own_gemm:
                self.lm_head = PackedWeight(self.lm_head)
            torch.cuda.synchronize(dev)
        self._device_index = self.x.get_device()
        self.parts = self._stream_parts() if streaming and 0 < b <= 16 else None

    def _fits(self, t: torch.Tensor, shape) -> bool:
        """``t`` is what the streamed kernels take an address for: bf16 rows of this shape on the step's device."""
        return t.shape == shape and t.dtype is torch.bfloat16 and t.get_device() == self._device_index \
            and t.is_contiguous() and not t.data_ptr() & 15

    def _layer_fits(self, L) -> bool:
        """The streamed kernels get addresses only.  Weights and caches may be replaced between steps, so this is asked
        on every step, like the checks of ``rope_append`` and ``torch.mm`` in the other form."""
        k = L["k"]
        cache = (self.x.shape[0], self.hkv, k.shape[2] if k.dim() == 4 else 0, self.d)
        if not self._fits(k, cache) or not self._fits(L["v"], cache):
            return False
        for name, shape in self._layer_shapes:
            if not self._fits(L[name], shape):
                return False
        return True

    def _ends_fit(self) -> bool:
        """The same for what the layers share."""
        b, hidden = self.x.shape
        lens, tables = self.seq_lens, (self.cos.shape[0], self.d)
        return (lens.dtype is torch.int32 and lens.numel() == b and lens.is_contiguous()
                and lens.get_device() == self._device_index and self._fits(self.cos, tables)
                and self._fits(self.sin, tables) and self._fits(self.final_norm, (hidden,))
                and self._fits(self.lm_head, (self.logits.shape[1], hidden)))

    def _stream_parts(self):
        """Scratch of the streamed projections (one buffer: each is consumed before the next is written), or None
        when a size or an address does not suit those kernels and the step stays on torch.mm, which refuses what is
        wrong rather than unsuitable."""
        hidden, inter = int(self.x.shape[1]), int(self.act.shape[1])
        if not self.x.is_cuda or hidden % 8 or hidden > 16384 or inter % 8 or self.d % 8:
            return None
        if not self._ends_fit() or not all(self._layer_fits(L) for L in self.layers):
            return None
        weights = [self.lm_head] + [L[n] for L in self.layers for n in ("w_qkv", "w_o", "w_gu", "w_down")]
        size = _lib.load().ia_llama_gemm_parts_bytes
        need = [int(size(int(w.shape[0]), int(w.shape[1]))) for w in weights]
        return torch.empty(max(need), dtype=torch.uint8, device=self.x.device) if min(need) > 0 else None

    def _linear(self, x: torch.Tensor, w, out: torch.Tensor) -> torch.Tensor:
        """nn.Linear without bias, where the projections are not streamed.  Back to back on its own, the
        packed-weight kernel matches cuBLAS at 32 rows and passes it on the widest shape (lm head, 6.6 against 6.5
        TB/s); inside the step its longer start-up and partial-tile tail cost about 7 us per projection, so it
        runs on request only."""
        if isinstance(w, PackedWeight):
            return gemm(x, w, out, self.gemm_ws)
        return torch.mm(x, w.t(), out=out)

    def _stream_step(self, tokens: torch.Tensor) -> bool:
        """The step with every projection streamed (``ia_llama_gemm_parts``): weights start to arrive while the kernel
        before still runs, and the element-wise kernels add up the partial sums.  False: something does not fit (any
        more), nothing that reads or writes it was launched, and the other form has to take the step from its start.
        Four full-size layers of Llama-3-8B at 7001 tokens, torch.mm / streamed, us: one sequence 746 / 674, 8 sequences
        811 / 754, 16 sequences 893 / 847."""
        if not self._ends_fit():
            return False
        lib, check, stream, b = _lib.load(), _lib.check, _stream(), self.x.shape[0]
        ctx_shape = (b, self.hq * self.d)
        parts, parts_bytes = self.parts.data_ptr(), self.parts.numel()
        x, h, q, act, hidden, inter = (self.x.data_ptr(), self.h.data_ptr(), self.q.data_ptr(), self.act.data_ptr(),
                                       self.x.shape[1], self.act.shape[1])
        cos, sin, max_pos, seq_lens = self.cos.data_ptr(), self.sin.data_ptr(), self.cos.shape[0], self.seq_lens.data_ptr()

        def gemm_parts(src, w, out=None):
            n, k = w.shape
            check(lib.ia_llama_gemm_parts(src, w.data_ptr(), out, b, n, k, parts, parts_bytes, stream))
            return k

        def add_norm(k, weight):
            check(lib.ia_llama_add_rmsnorm_parts(x, parts, k, weight.data_ptr(), h, b, hidden, self.eps, stream))

        k = None
        for L, attn in zip(self.layers, self.attention):
            if not self._layer_fits(L):
                return False
            if k is None:
                add_rmsnorm(self.x, None, L["norm1"], self.eps, self.h)
            else:
                add_norm(k, L["norm1"])
            k = gemm_parts(h, L["w_qkv"])
            k_cache, v_cache = L["k"], L["v"]
            t = k_cache.shape[2]
            check(lib.ia_llama_rope_append_parts(parts, k, cos, sin, max_pos, seq_lens, k_cache.data_ptr(),
                                                 v_cache.data_ptr(), self.hkv * t * self.d, t * self.d, t, q, b, self.hq,
                                                 self.hkv, self.d, stream))
            ctx = attn.step(self.q).view(ctx_shape)
            if not self._fits(ctx, ctx_shape):
                return False
            k = gemm_parts(ctx.data_ptr(), L["w_o"])
            add_norm(k, L["norm2"])
            k = gemm_parts(h, L["w_gu"])
            check(lib.ia_llama_silu_mul_parts(parts, k, act, b, inter, stream))
            k = gemm_parts(act, L["w_down"])
        if k is None:
            add_rmsnorm(self.x, None, self.final_norm, self.eps, self.h)
        else:
            add_norm(k, self.final_norm)
        k = gemm_parts(h, self.lm_head, self.logits.data_ptr())
        check(lib.ia_llama_argmax_parts(parts, k, self.logits.data_ptr(), b, self.logits.shape[1], tokens.data_ptr(), stream))
        return True

    @torch.no_grad()
    def step(self, tokens: torch.Tensor) -> torch.Tensor:
        if self.parts is not None and tokens.device == self.x.device and tokens.dtype == torch.int64 \
                and tokens.is_contiguous() and tokens.numel() == self.x.shape[0]:
            torch.index_select(self.embed, 0, tokens.view(-1), out=self.x)
            if self._stream_step(tokens):
                return tokens
        b = self.x.shape[0]
        torch.index_select(self.embed, 0, tokens.view(-1), out=self.x)
        delta = None
        for L, attn in zip(self.layers, self.attention):
            add_rmsnorm(self.x, delta, L["norm1"], self.eps, self.h)
            self._linear(self.h, L["w_qkv"], self.qkv)
            rope_append(self.qkv, self.cos, self.sin, self.seq_lens, L["k"], L["v"], self.q)
            ctx = attn.step(self.q)
            self._linear(ctx.view(b, self.hq * self.d), L["w_o"], self.o)
            add_rmsnorm(self.x, self.o, L["norm2"], self.eps, self.h)
            self._linear(self.h, L["w_gu"], self.gu)
            silu_mul(self.gu, self.act)
            self._linear(self.act, L["w_down"], self.down)
            delta = self.down
        add_rmsnorm(self.x, delta, self.final_norm, self.eps, self.h)
        self._linear(self.h, self.lm_head, self.logits)
        argmax(self.logits, tokens)
        return tokens
