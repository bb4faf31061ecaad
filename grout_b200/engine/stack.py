"""A decode step's layers as one kernel (``csrc/decode_stack.cu``), for models whose layers it knows.

The kernel runs a plain pre-norm decoder layer: RMS norms, grouped-query attention over the whole
paged cache with 128-wide heads (with or without the heads' norms, the whole head rotated), a
gated SiLU feed-forward, bfloat16 weights.  ``stack_layers`` says whether a model is that, layer
by layer and attribute by attribute; anything else (a window, a cap, a bias, a part of the
caller's own, 32-bit weights, another product kernel or a decode attention asked for) goes layer
by layer as before."""
from __future__ import annotations

import weakref
from typing import List, Optional

import torch

from ..kernels import ops
from ..parts.block import PreNormBlock
from ..parts.feedforward import SwiGLU
from ..parts.linear import Linear
from ..parts.mixer import GQAAttention
from ..parts.norm import RMSNorm
from ..parts.position import RotaryHalfSplit

HEAD = 128

# Up to how many keys a step of so many (sequence, kv head) pairs goes to the kernel; (the most pairs, the most keys).
# The kernel divides a pair's keys into units that are a block's whole work, one block an SM, so with many pairs a long
# sequence among short ones is cut into few units and most blocks wait for its: with 16 kv heads one of 32,768 keys
# beside seven of 100 is two units a head.  Measured on 148 SMs, captured steps, us a step by this kernel / layer by
# layer, the worst of all ways to mix long sequences with short ones, at the sizes (hidden, kv heads, feed-forward,
# layers) where layer by layer does best:
#   up to 32 pairs    4 sequences of 39,000 keys (4096, 8, 12288, 12) 2,052 / 2,324; 1 of 4,000 (4096, 20, 12288, 8) 742 / 783
#   up to 64 pairs    5 of 4,000 and 2 of 100 (4096, 9, 12288, 8) 833 / 832, 8 of 2,000 (4096, 8, 12288, 12) 1,140 / 1,175;
#                     but 6 of 12,000 and 2 of 100 (the same) 1,588 / 1,572, 6 of 32,000 and 2 of 100 2,581 / 2,411
#   up to 128 pairs   3 of 1,010 and 5 of 100 (4096, 12, 12288, 8) 751 / 753; but 2 of 2,000 and 6 of 100
#                     (4096, 16, 12288, 8) 818 / 797, 2 of 32,000 and 6 of 100 2,923 / 2,019
#   more              2 of 500 and 6 of 100 (4096, 20, 12288, 8) 770 / 773; but 1 of 1,010 and 7 of 100 807 / 802, 1 of
#                     32,000 and 7 of 100 (3072, 24, 8192, 8) 2,767 / 1,087
KEYS_MOST = ((32, None), (64, 4096), (128, 1024), (None, 512))


#: What the kernel does in place of these; where one has been replaced (to look at what a layer does, for instance),
#: in its class or on one object, layers run one by one.
_DONE = {PreNormBlock: ("forward",), GQAAttention: ("forward", "_attend"), SwiGLU: ("forward",),
         RMSNorm: ("add_norm", "forward"), RotaryHalfSplit: ("rotary",), Linear: ("__call__", "silu_mul")}
_METHODS = tuple((cls, name, getattr(cls, name)) for cls, names in _DONE.items() for name in names)


def _as_it_is(x) -> bool:
    return vars(x).keys().isdisjoint(_DONE[type(x)])


def _plain_linear(lin, out_features: int, in_features: int) -> bool:
    return (type(lin) is Linear and _as_it_is(lin) and lin.weight.dtype == torch.bfloat16 and lin.decode_kernel == "tc"
            and lin.weight.is_contiguous() and tuple(lin.weight.shape) == (out_features, in_features)
            and lin.weight.data_ptr() % 16 == 0)


def _plain_weights(w, width: int) -> bool:
    """A norm's weights as the kernel reads them: in pieces of 16 bytes, 32-bit or bfloat16."""
    return (isinstance(w, torch.Tensor) and tuple(w.shape) == (width,) and w.dtype in (torch.float32, torch.bfloat16)
            and w.is_contiguous() and w.data_ptr() % 16 == 0)


def _plain_norm(norm, width: int) -> bool:
    return type(norm) is RMSNorm and _as_it_is(norm) and _plain_weights(norm.weight, width)


def _plain_rotation(position) -> bool:
    if type(position) is not RotaryHalfSplit or not _as_it_is(position):
        return False
    rot = position.rotary()
    return (rot.rot_dim == HEAD and not rot.interleaved and rot.amplitude == 1.0 and rot.inv_freq.is_contiguous()
            and rot.inv_freq.dtype == torch.float32)


def _plain_attention(m) -> bool:
    return (type(m) is GQAAttention and _as_it_is(m) and m.D == m.Dv == m.Ds == HEAD and _plain_rotation(m.position)
            and m.window is None and not m.chunk and not m.keep_first and m.softcap is None and m.sink is None
            and not m.head_gate and not m.beside and not m.shares_kv and not m.values_are_keys
            and not m.conv_path and m.taps == 1 and m.q_temp is None
            and all(w is None if m.qk_norm_eps is None else _plain_weights(w, HEAD) for w in (m.q_norm_w, m.k_norm_w))
            and _plain_linear(m.qkv, (m.nq + 2 * m.nkv) * HEAD, m.hidden) and _plain_linear(m.o, m.hidden, m.nq * HEAD))


def _plain_layer(block) -> bool:
    if (type(block) is not PreNormBlock or not _as_it_is(block) or type(block.feedforward) is not SwiGLU
            or not _as_it_is(block.feedforward) or not _plain_attention(block.mixer)):
        return False
    m, f = block.mixer, block.feedforward
    return (f.interleave == 8 and f.hidden == m.hidden and _plain_linear(f.gate_up, 2 * f.intermediate, f.hidden)
            and _plain_linear(f.down, f.hidden, f.intermediate)
            and _plain_norm(block.norm1, m.hidden) and _plain_norm(block.norm2, m.hidden))


def _sizes(block):
    m = block.mixer
    return (m.hidden, block.feedforward.intermediate, m.nq, m.nkv, m.scale, m.qk_norm_eps, block.norm1.eps,
            block.norm2.eps)


def stack_layers(model) -> Optional[List]:
    """The model's blocks in the order they run when the kernel can run all of them, else None (as soon as one is found
    that it cannot: every decode step that is not replayed asks)."""
    if model.ctx.dtype != torch.bfloat16 or any(getattr(cls, name) is not f for cls, name, f in _METHODS):
        return None
    blocks = []
    for e in model.plan.schedule:
        block = model.blocks[e.layer]
        if (e.cache_of is not None or e.add is not None or e.average is not None or not _plain_layer(block)
                or (blocks and _sizes(block) != _sizes(blocks[0]))):
            return None
        blocks.append(block)
    return blocks if blocks and blocks[0].norm1.eps == blocks[0].norm2.eps else None


def _made_from(blocks) -> tuple:
    """What a ``DecodeStack`` takes from the layers: their sizes and constants, where the weights lie, which the kernel
    reads there at every launch, and the rotations' tables, of which it reads the first layer's."""
    out = [_sizes(blocks[0])]
    for b in blocks:
        m, f, freq = b.mixer, b.feedforward, b.mixer.position.rotary().inv_freq
        out.append(tuple(lin.weight.data_ptr() for lin in (m.qkv, m.o, f.gate_up, f.down)))
        out.append(tuple((w.data_ptr(), w.dtype) for w in (b.norm1.weight, b.norm2.weight, m.q_norm_w, m.k_norm_w)
                         if w is not None))
        out.append((freq.data_ptr(), 0 if freq.is_inference() else freq._version))
    return tuple(out)


class DecodeStack:
    """The kernel's view of one model and one cache: every layer's tensor maps and vectors on the
    device, and the scratch of its launches, which are ordered on one stream as the steps of an
    engine are."""

    def __init__(self, blocks, views, max_rows: int = ops.DECODE_STACK_ROWS):
        hidden, ff, nq, nkv, scale, qk_eps, eps, _eps = _sizes(blocks[0])
        device = blocks[0].mixer.qkv.weight.device
        self.hidden, self.nkv, self.max_rows = hidden, nkv, max_rows
        self._layers = []                 # (the tensors that the device's table points at)
        for b, view in zip(blocks, views):
            m, f = b.mixer, b.feedforward
            self._layers.append(dict(
                qkv=m.qkv.weight, o=m.o.weight, gate_up=f.gate_up.weight, down=f.down.weight, k_pages=view.k_pages,
                v_pages=view.v_pages, norm1=b.norm1.weight, norm2=b.norm2.weight, q_norm=m.q_norm_w, k_norm=m.k_norm_w))
        self.block_table = views[0].block_table
        self.state = ops.decode_stack_state(self._layers, hidden, ff, nq, nkv, max_rows, device)
        self.args = dict(eps=eps, qk_eps=qk_eps or 0.0, scale=scale,
                         inv_freq=blocks[0].mixer.position.rotary().inv_freq)

    @classmethod
    def of(cls, blocks, cache) -> Optional["DecodeStack"]:
        """None when the cache is not one that the kernel reads, the layers rotate differently or their sizes have no plan."""
        views = [cache.view(i) for i in range(len(blocks))]
        table = views[0].block_table
        for b, v in zip(blocks, views):
            if (v.page != 64 or v.k_pages.dtype != torch.bfloat16 or v.block_table.data_ptr() != table.data_ptr()
                    or tuple(v.k_pages.shape[1:]) != (b.mixer.nkv, 64, HEAD) or v.v_pages.shape != v.k_pages.shape
                    or v.k_pages.data_ptr() == v.v_pages.data_ptr()):
                return None
        freq = blocks[0].mixer.position.rotary().inv_freq
        if not all(torch.equal(b.mixer.position.rotary().inv_freq, freq) for b in blocks[1:]):
            return None
        hidden, ff, nq, nkv = _sizes(blocks[0])[:4]
        if not ops.decode_stack_takes(hidden, ff, nq, nkv, table.device):
            return None
        return cls(blocks, views)

    def takes(self, step) -> bool:
        """Whether the step is one that the kernel runs, and runs faster: decided by what a captured step is bounded by."""
        if not step.decode or not 0 < step.n_tokens <= self.max_rows or step.n_seqs != step.n_tokens:
            return False
        keys = next(keys for pairs, keys in KEYS_MOST if pairs is None or step.n_tokens * self.nkv <= pairs)
        return keys is None or step.max_kv_len <= keys

    def reads(self, res, pending) -> bool:
        """Whether the kernel reads what stands in front of the layers: the 32-bit stream or its first contribution in
        bfloat16, as this library's embeddings leave it (a caller's own may leave something else)."""
        x = pending if res is None else res
        return ((res is None or pending is None) and isinstance(x, torch.Tensor) and x.dim() == 2
                and x.shape[1] == self.hidden and x.is_contiguous()
                and x.dtype == (torch.bfloat16 if res is None else torch.float32))

    def forward(self, res, pending, step) -> torch.Tensor:
        """The 32-bit stream behind the last layer, [T, hidden]."""
        return ops.decode_stack(self.state, res, pending, slots=step.slots, kv_len=step.kv_len,
                                block_table=self.block_table, **self.args)


class StackOf:
    """A model's ``DecodeStack``s, one for each cache that its steps use, made anew when what they take from the layers has
    changed (steps that are replayed from a captured graph do not come here: they run what was there at the capture).
    They hold the caches' pages, so they go with their caches."""

    def __init__(self):
        self._stacks = weakref.WeakKeyDictionary()       # cache -> (what it was made from, stack)

    def clear(self) -> None:
        """Lets go of the weights and pages that the stacks hold."""
        self._stacks.clear()

    def get(self, model, cache) -> Optional[DecodeStack]:
        if ops.DECODE_ATTENTION != "auto" or ops.DECODE_SPLITS_OVERRIDE or ops.DECODE_TMA_STAGES:
            return None                  # (a kernel, or its division of the keys, is asked for)
        blocks = stack_layers(model)
        if blocks is None:
            return None
        made_from = _made_from(blocks)
        known, stack = self._stacks.get(cache, (None, None))
        if known != made_from:
            if torch.cuda.is_available() and torch.cuda.is_current_stream_capturing():
                return None              # (it takes copies and comparisons that the host waits for)
            self._stacks.pop(cache, None)
            stack = DecodeStack.of(blocks, cache)
            self._stacks[cache] = (made_from, stack)
        return stack
