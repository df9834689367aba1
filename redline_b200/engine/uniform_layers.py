"""Models whose layers are all alike, for the paths that take a whole step at once."""

from __future__ import annotations

from operator import attrgetter
from typing import List, Optional

import torch

from ..parts.attention import GQAttention
from ..parts.block import PreNormBlock
from ..parts.mlp import SwiGLUMLP
from ..parts.rmsnorm import RMSNorm


# What a step runs of a block and its parts.
_METHODS = attrgetter("forward", "mixer.forward", "mixer.forward_into", "ffn.forward", "ffn.forward_into", "mixer_norm.add_norm",
                      "ffn_norm.add_norm")
_CLASS_METHODS = (PreNormBlock.forward, GQAttention.forward, GQAttention.forward_into, SwiGLUMLP.forward, SwiGLUMLP.forward_into,
                  RMSNorm.add_norm, RMSNorm.add_norm)


def uniform_layers(model, caches: List[object]) -> Optional[list]:
    """The blocks in run order if every one is a pre-norm block of RMSNorm, grouped-query attention with rotary tables
    and a SiLU-gated feed-forward of the same sizes, bfloat16 and without biases, that writes a cache of its own in the
    same group; None otherwise, and where one of them has a method of its own (a wrapper around ``forward``, say)."""
    rt, order = model.rt, model.spec.order
    if rt.dtype != torch.bfloat16 or not order:
        return None
    blocks = [model.blocks[call.layer] for call in order]
    first = blocks[0]
    for call, b, cache in zip(order, blocks, caches):
        if (type(b) is not PreNormBlock or type(b.mixer) is not GQAttention or type(b.ffn) is not SwiGLUMLP
                or type(b.mixer_norm) is not RMSNorm or type(b.ffn_norm) is not RMSNorm or call.add_embedding
                or cache is None or not cache.write or cache.group != caches[0].group or not b.ffn.silu):
            return None
        if any(getattr(m, "__func__", None) is not of_class for m, of_class in zip(_METHODS(b), _CLASS_METHODS)):
            return None
        att, ffn, a0, f0 = b.mixer, b.ffn, first.mixer, first.ffn
        if any(t is not None for t in (att.b_qkv, att.b_o, ffn.b_gate_up, ffn.b_down)):
            return None
        if (att.params != a0.params or att.scale != a0.scale or ffn.params != f0.params
                or ffn.params.hidden_size != att.params.hidden_size or att.position.rotary_tables() is None):
            return None
        tensors = [att.w_qkv, att.w_o, ffn.w_gate_up, ffn.w_down, b.mixer_norm.weight, b.ffn_norm.weight, cache.k, cache.v]
        if any(t.dtype != torch.bfloat16 or not t.is_contiguous() or t.data_ptr() % 16 for t in tensors):
            return None
        if {b.mixer_norm.params.eps, b.ffn_norm.params.eps} != {first.mixer_norm.params.eps}:
            return None
    return blocks
