"""Which decode steps run their layers as one kernel, and how long what they read lives: on the host, with the kernel's
state replaced by a stand-in."""
import gc
import weakref

import pytest
import torch

from grout_b200.config import resolve_architecture
from grout_b200.engine import stack
from grout_b200.engine.graphs import StepGraph
from grout_b200.engine.model import Model
from grout_b200.kernels import ops
from grout_b200.parts.base import BuildContext
from grout_b200.weights import random_tensor

CONFIG = dict(architectures=["Qwen3ForCausalLM"], model_type="qwen3", vocab_size=64, hidden_size=256, intermediate_size=192,
              num_hidden_layers=3, num_attention_heads=2, num_key_value_heads=1, head_dim=128, rope_theta=1000000.0,
              rms_norm_eps=1e-6, max_position_embeddings=512, tie_word_embeddings=True, use_sliding_window=False,
              eos_token_id=63)


class Cache:
    """Something that a model's steps use and that can be referred to weakly."""


class Made:
    """What stands in for the kernel's state."""


def load(config=CONFIG, dtype=torch.bfloat16):
    arch = resolve_architecture(config)
    model = Model(arch.plan(arch.config_cls.from_dict(config)), BuildContext(dtype, torch.device("cpu")))
    expected = model.expected()
    model.load(lambda name: random_tensor(name, expected[name], 1, dtype, torch.device("cpu")))
    return model


@pytest.fixture
def model(monkeypatch):
    monkeypatch.setattr(stack.DecodeStack, "of", classmethod(lambda cls, *args: Made()))
    return load()


def captured(model, cache):
    """A decode graph as far as it goes without a GPU."""
    g = StepGraph.__new__(StepGraph)
    g.model, g.cache, g.decode = model, cache, True
    g._hold()
    return g


def test_a_captured_step_keeps_what_it_was_captured_with(model):
    cache = Cache()
    g = captured(model, cache)
    seen = weakref.ref(g.holds)
    norm = model.blocks[1].norm2
    norm.weight = norm.weight.clone()
    assert model.decode_stack(cache) is not g.holds      # made anew for the other weight
    gc.collect()
    assert seen() is not None
    del g
    gc.collect()
    assert seen() is None


def test_weights_made_in_inference_mode(model):
    """They have no version counter; a model that the kernel does not take is asked about like any other."""
    with torch.inference_mode():
        m, cache = load(), Cache()
        assert isinstance(m.decode_stack(cache), Made) and m.decode_stack(cache) is m.decode_stack(cache)
        assert load(dict(CONFIG, head_dim=64)).decode_stack(cache) is None


@pytest.mark.parametrize("name,value", [("DECODE_ATTENTION", "tma"), ("DECODE_ATTENTION", "mma"),
                                        ("DECODE_SPLITS_OVERRIDE", 4), ("DECODE_TMA_STAGES", 3)])
def test_a_decode_attention_that_is_asked_for_is_taken(model, monkeypatch, name, value):
    cache = Cache()
    assert model.decode_stack(cache) is not None
    monkeypatch.setattr(ops, name, value)
    assert model.decode_stack(cache) is None


CHANGES = {
    "a window": lambda b: setattr(b.mixer, "window", 64),
    "a softcap": lambda b: setattr(b.mixer, "softcap", 30.0),
    "a query temperature": lambda b: setattr(b.mixer, "q_temp", (0.1, 64)),
    "a scale": lambda b: setattr(b.mixer, "scale", 0.5),
    "an epsilon": lambda b: setattr(b.norm2, "eps", 1e-3),
    "another product kernel": lambda b: setattr(b.feedforward.down, "decode_kernel", "skinny"),
    "a weight that is not contiguous": lambda b: setattr(b.mixer.o, "weight", b.mixer.o.weight.t().contiguous().t()),
    "a norm at an odd place": lambda b: setattr(b.norm1, "weight", torch.ones(257, dtype=torch.bfloat16)[1:]),
    "a mixer that is looked at": lambda b: setattr(b.mixer, "forward", lambda *a: type(b.mixer).forward(b.mixer, *a)),
    "a product that is looked at": lambda b: setattr(b.feedforward.gate_up, "silu_mul", lambda *a: None),
}


@pytest.mark.parametrize("change", CHANGES)
def test_layers_that_change_after_the_first_step_run_one_by_one(model, change):
    """A step that is not replayed reads what the layers are then, as it does without the kernel."""
    cache = Cache()
    assert model.decode_stack(cache) is not None
    CHANGES[change](model.blocks[1])
    assert model.decode_stack(cache) is None


def test_what_all_layers_share_may_change(model):
    cache = Cache()
    a = model.decode_stack(cache)
    for b in model.blocks:
        b.mixer.scale = 0.5
    b = model.decode_stack(cache)
    assert b is not None and b is not a and model.decode_stack(cache) is b
    model.blocks[0].mixer.position.rotary().inv_freq.mul_(0.5)       # (what it is is compared when the state is made)
    assert model.decode_stack(cache) is not b


def test_a_class_whose_method_is_replaced(model, monkeypatch):
    cache, mixer = Cache(), type(model.blocks[0].mixer)
    assert model.decode_stack(cache) is not None
    was = mixer.forward
    monkeypatch.setattr(mixer, "forward", lambda self, *a: was(self, *a))
    assert model.decode_stack(cache) is None


def test_a_stack_goes_with_its_cache(monkeypatch):
    """It holds the cache's pages; and two engines over one model do not take turns at one stack."""
    def made(cls, blocks, cache):
        out = Made()
        out.pages = cache.pages
        return out
    monkeypatch.setattr(stack.DecodeStack, "of", classmethod(made))
    model, caches = load(), [Cache(), Cache()]
    for c in caches:
        c.pages = Made()
    stacks = [model.decode_stack(c) for c in caches]
    assert stacks[0] is not stacks[1] and [model.decode_stack(c) for c in caches] == stacks
    pages = weakref.ref(caches[0].pages)
    del stacks, c
    caches.pop(0)
    gc.collect()
    assert pages() is None


def test_other_tensors_are_loaded(model):
    """The tensors that were there before are not kept until the next step."""
    cache = Cache()
    held = weakref.ref(model.decode_stack(cache))
    expected = model.expected()
    model.load(lambda name: random_tensor(name, expected[name], 2, torch.bfloat16, torch.device("cpu")))
    gc.collect()
    assert held() is None


def bare_stack(monkeypatch, nkv=1):
    monkeypatch.setattr(ops, "decode_stack_state", lambda *args: None)
    view = type("View", (), {"k_pages": None, "v_pages": None, "block_table": None})
    return stack.DecodeStack(load(dict(CONFIG, num_attention_heads=nkv, num_key_value_heads=nkv)).blocks, [view] * 3)


def test_what_stands_in_front_of_the_layers(monkeypatch):
    """A caller's own embedding may leave partial sums, a wider type or a ``Contribution``; the norms take them all."""
    from grout_b200.parts.norm import Contribution
    st = bare_stack(monkeypatch)
    narrow, wide = torch.zeros((2, 256), dtype=torch.bfloat16), torch.zeros((2, 256))
    assert st.reads(None, narrow) and st.reads(wide, None)
    for res, pending in ((None, wide), (narrow, None), (wide, narrow), (None, None), (None, wide[None].expand(3, 2, 256)),
                         (None, Contribution(narrow)), (None, narrow.t().contiguous().t())):
        assert not st.reads(res, pending)


@pytest.mark.parametrize("nkv,rows,most", [(8, 1, 1 << 20), (8, 4, 1 << 20), (32, 1, 1 << 20), (8, 5, 4096), (8, 8, 4096),
                                           (16, 4, 4096), (16, 5, 1024), (16, 8, 1024), (17, 8, 512), (32, 8, 512)])
def test_as_many_keys_as_the_kernel_is_faster_with(monkeypatch, nkv, rows, most):
    st = bare_stack(monkeypatch, nkv)
    step = type("Step", (), dict(decode=True, n_tokens=rows, n_seqs=rows, max_kv_len=most))
    assert st.takes(step)
    step.max_kv_len = most + 1
    assert st.takes(step) is (rows * nkv <= 32)
    step.max_kv_len, step.decode = 1, False
    assert not st.takes(step)
