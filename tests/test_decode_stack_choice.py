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
    monkeypatch.setattr(stack.DecodeStack, "of", classmethod(lambda cls, model, cache: Made()))
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
        for config in (CONFIG, dict(CONFIG, head_dim=64)):
            m, cache = load(config), Cache()
            assert isinstance(m.decode_stack(cache), Made) and m.decode_stack(cache) is m.decode_stack(cache)


@pytest.mark.parametrize("name,value", [("DECODE_ATTENTION", "tma"), ("DECODE_ATTENTION", "mma"),
                                        ("DECODE_SPLITS_OVERRIDE", 4), ("DECODE_TMA_STAGES", 3)])
def test_a_decode_attention_that_is_asked_for_is_taken(model, monkeypatch, name, value):
    cache = Cache()
    assert model.decode_stack(cache) is not None
    monkeypatch.setattr(ops, name, value)
    assert model.decode_stack(cache) is None
