"""Models whose layers are all alike, for the paths that take a whole step at once."""

from __future__ import annotations

from functools import lru_cache
from inspect import isfunction
from typing import List, Optional

import torch

from ..parts.attention import GQAttention
from ..parts.block import PreNormBlock
from ..parts.mlp import SwiGLUMLP
from ..parts.rmsnorm import RMSNorm


@lru_cache(maxsize=None)
def _methods(kind: type) -> tuple:
    found = {}
    for k in reversed(kind.__mro__):
        found.update((name, f) for name, f in vars(k).items() if isfunction(f))
    return tuple(found.items())


def _own_method(part) -> bool:
    """Whether the object has a method of its own in place of its class's (a wrapper around ``forward``, say).  (Asked by
    attribute: a look into an object's ``__dict__`` would make its attributes slower for good.)"""
    return any(getattr(getattr(part, name), "__func__", None) is not f for name, f in _methods(type(part)))


def uniform_layers(model, caches: List[object]) -> Optional[list]:
    """The blocks in run order if every one is a pre-norm block of RMSNorm, grouped-query attention with rotary tables
    and a SiLU-gated feed-forward of the same sizes, bfloat16 and without biases, that writes a cache of its own in the
    same group; None otherwise, and where one of them has a method of its own."""
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
        if any(map(_own_method, (b, b.mixer, b.mixer.position, b.ffn, b.mixer_norm, b.ffn_norm))):
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
