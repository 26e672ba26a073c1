"""Host-side behaviour of the reference-named calls, without a GPU: tensors that only claim to be on one (fake
tensors), and a library that records its calls instead of launching anything."""

import copy
import io

import pytest
import torch
from torch._subclasses.fake_tensor import FakeTensorMode

from interattn_b200 import _lib, ops, reference_api as api

HKV, G, D, BLOCK, PROMPT = 2, 4, 64, 64, 128
NB = PROMPT // BLOCK


def _prefix(device):
    new = lambda *shape, dtype=torch.bfloat16: torch.empty(shape, dtype=dtype, device=device)  # noqa: E731
    cache = [new(HKV, PROMPT + 64, D)[:, :PROMPT] for _ in range(2)]
    slab = (1, HKV, NB, D)
    summ = ops.BlockSummaries(k_bar=new(*slab, dtype=torch.float32), k_max=new(*slab), k_min=new(*slab),
                              v_bar=new(*slab), v_norm_max=new(1, HKV, NB, dtype=torch.float32), block_size=BLOCK)
    geometry = api._CacheGeometry(device, PROMPT)
    return {"block_valid_counts": new(NB, dtype=torch.int64),
            "_b200": api._PrefixHandle(*cache, BLOCK, summ, geometry)}


@pytest.mark.filterwarnings("ignore:Accessing the data pointer")
def test_the_suffix_length_lives_on_the_cache_device():
    """The kernels read the length where it lies, so a scalar of another GPU is refused and not dereferenced."""
    with FakeTensorMode():
        prefix = _prefix("cuda:0")
        q = torch.empty((HKV, G, 1, D), dtype=torch.bfloat16, device="cuda:0")
        empty = torch.empty((HKV, 0, D), dtype=torch.bfloat16, device="cuda:0")
        for length in (torch.zeros((), dtype=torch.int32, device="cuda:1"), torch.zeros((1,), dtype=torch.int64, device="cuda:1"),
                       torch.zeros((), dtype=torch.int32)):
            with pytest.raises(ValueError, match="suffix_len_dev"):
                api._condition_block_decode_output_fused_triton(
                    q_grouped=q, prompt_prefix=prefix, k_suffix=empty, v_suffix=empty, suffix_len_dev=length, eps=None,
                    top_k=1, page_size=BLOCK, store_selected=False, output_dtype=None, workspace={})


def _pointers(struct):
    return [getattr(struct, name) for name, _ in struct._fields_]


@pytest.mark.parametrize("how", ["copy", "deepcopy", "save"])
def test_a_prefix_can_be_copied_and_saved(how):
    """The handle keeps the summaries' addresses in the form the library takes; a copy has those of its own tensors."""
    prefix = _prefix("cpu")
    prefix["_b200"].summ.v_bar.fill_(3.0)
    if how == "save":
        buf = io.BytesIO()
        torch.save(prefix, buf)
        buf.seek(0)
        other = torch.load(buf, weights_only=False)
    else:
        other = getattr(copy, how)(prefix)
        if how == "copy":
            other["_b200"] = copy.copy(prefix["_b200"])
    h = other["_b200"]
    assert _pointers(h.c_summ) == _pointers(h.summ.c_struct())
    assert (_pointers(h.c_summ) == _pointers(prefix["_b200"].c_summ)) == (how == "copy")
    assert torch.equal(h.summ.v_bar, prefix["_b200"].summ.v_bar)
    assert (h.block_size, h.prompt_len, h.geom_flags) == (BLOCK, PROMPT, prefix["_b200"].geom_flags)


class _Library:
    """Takes any call and remembers its name."""

    def __init__(self):
        self.calls = []

    def __getattr__(self, name):
        def call(*args):
            self.calls.append(name)
            return 0
        return call


@pytest.fixture
def recorder(monkeypatch):
    lib = _Library()
    monkeypatch.setattr(api._lib, "load", lambda: lib)
    monkeypatch.setattr(api, "_stream", lambda: None)
    return lib


@pytest.mark.filterwarnings("ignore:Accessing the data pointer")
@pytest.mark.parametrize("length", [PROMPT - 1, PROMPT])
@pytest.mark.parametrize("which", ["k", "v"])
def test_blocked_copies_carry_a_tangent(length, which, recorder):
    """Forward-mode differentiation goes through k_block_attn / v_block_attn, padded copies or views alike."""
    from torch.autograd import forward_ad
    with FakeTensorMode(), forward_ad.dual_level():
        k, v = (torch.empty((HKV, length, D), dtype=torch.bfloat16, device="cuda:0") for _ in range(2))
        dual = forward_ad.make_dual(k if which == "k" else v, torch.empty_like(k))
        prefix = api._build_prompt_blocks(dual if which == "k" else k, dual if which == "v" else v, BLOCK)
        assert recorder.calls == ["ia_build_prompt_blocks"]
        for name in ("k", "v"):
            tangent = forward_ad.unpack_dual(prefix[f"{name}_block_attn"]).tangent
            assert (tangent is not None) == (name == which), name


@pytest.mark.filterwarnings("ignore:Accessing the data pointer")
def test_blocked_copies_of_a_cache_with_gradients(recorder):
    with FakeTensorMode():
        k, v = (torch.empty((HKV, PROMPT - 1, D), dtype=torch.bfloat16, device="cuda:0") for _ in range(2))
        assert api._build_prompt_blocks(k, v.requires_grad_(), BLOCK)["v_block_attn"].requires_grad


@pytest.mark.parametrize("mixed", ["0", "1"])
@pytest.mark.parametrize("packed", ["0", "1"])
@pytest.mark.filterwarnings("ignore:Accessing the data pointer")
def test_every_array_of_a_prefix_has_its_own_storage(packed, mixed, recorder, monkeypatch):
    """Keeping, saving or changing one of them does not keep, save or touch another (the views into the packed
    range apart)."""
    monkeypatch.setenv("CONDITION_BLOCK_TMA_BOUNDS", packed)
    monkeypatch.setenv("CONDITION_BLOCK_MIXED_SUMMARIES", mixed)
    with FakeTensorMode():
        k, v = (torch.empty((HKV, PROMPT - 1, D), dtype=torch.bfloat16, device="cuda:0") for _ in range(2))
        prefix = api._build_prompt_blocks(k, v, BLOCK)
    views = {"k_max", "k_min"} if packed == "1" else set()
    for name, t in prefix.items():
        if torch.is_tensor(t) and name not in views:
            assert t.untyped_storage().nbytes() == t.numel() * t.element_size(), name
            assert t.is_contiguous() and (t._base is None or t._base.numel() == t.numel()), name
    h = prefix["_b200"]
    stored = [h.summ.k_bar, h.summ.v_bar, h.summ.v_norm_max] + ([h.summ.k_bounds] if views else [h.summ.k_max, h.summ.k_min])
    assert all(t.untyped_storage().nbytes() == t.numel() * t.element_size() for t in stored)
    if views:
        assert all(getattr(h.summ, n).shape == (1, HKV, NB, D) and getattr(h.summ, n).stride(3) == 2 for n in views)
        assert h.summ.k_min.storage_offset() == h.summ.k_bounds.storage_offset() + 1
