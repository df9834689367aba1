"""The layers of a prompt step, launched from native code (csrc/prompt_layers.cpp).

For models whose layers are all alike (``uniform_layers``): the same kernels with the same arguments as the parts launch
one by one, without Python between them.  Steps of 17 rows and more that hold a portion of some prompt; smaller ones,
steps of single tokens, profiled steps and steps that keep their sums in float32 go through the parts.
"""

from __future__ import annotations

import ctypes
import os
import warnings
from ctypes import c_float, c_int, c_int32, c_longlong, c_void_p
from operator import is_
from typing import List, Optional

import torch

from ..ops import kernels
from ..parts.base import Watched
from ..parts.mlp import TC_MIN_ROWS
from .uniform_layers import uniform_layers


class _Layer(ctypes.Structure):
    _fields_ = [(n, c_void_p) for n in ("w_qkv", "w_o", "w_gate_up", "w_down", "norm_mixer", "norm_ffn", "kcache", "vcache",
                                        "counters")]


class _Plan(ctypes.Structure):
    _fields_ = [(n, c_void_p) for n in (
        "gemm_ex", "set_math_mode", "add_rmsnorm", "rope", "attn_decode", "attn_prefill", "gemm_tc", "gemm_mid", "swiglu",
        "layers", "residual", "normed", "qkv", "attn", "mixer_out", "act", "gate_up", "ffn_out", "hand_xw_a", "hand_xw_b",
        "hand_sums_a", "hand_sums_b", "part_o", "part_ml", "cos", "sin", "status", "tc_status")]
    _fields_ += [("num_slots", c_longlong), ("eps", c_float), ("scale", c_float)]
    _fields_ += [(n, c_int32) for n in ("num_layers", "H", "I", "hq", "hkv", "D", "page_size", "window", "max_pos", "sm_count",
                                        "tc_min_rows", "hand_tiles")]


class _Step(ctypes.Structure):
    _fields_ = [(n, c_void_p) for n in ("blas", "stream", "positions", "slots", "block_table", "decode_info", "tile_seq",
                                        "tile_tok", "tile_rows")]
    _fields_ += [(n, c_int32) for n in ("T", "max_blocks", "num_decode", "decode_parts", "num_tiles", "decode_impl")]


class _Counts(ctypes.Structure):
    _fields_ = [("launches", c_int32), ("failed", c_int32)]


# The plan's launchers by the names that their errors have elsewhere.
_LAUNCHERS = ("cublasGemmEx", "cublasSetMathMode", "add_rmsnorm", "rope_kv_write", "attn_decode", "attn_prefill", "gemm_tc",
              "gemm_mid", "swiglu")


def _library(name: str):
    """A function of the cuBLAS that torch has loaded, or None, with a warning (torch without it)."""
    soname = f"libcublas.so.{(torch.version.cuda or '').split('.')[0]}"
    try:
        return getattr(ctypes.CDLL(soname, mode=os.RTLD_NOLOAD | os.RTLD_NOW), name)
    except (OSError, AttributeError):
        warnings.warn(f"{soname} is not loaded or has no {name}: the layers of prompt steps are launched from Python")
        return None


class PromptLayers:
    @staticmethod
    def of(model, caches: List[object], ctx) -> Optional["PromptLayers"]:
        """The plan for this model with these caches, or None if its layers are not alike."""
        blocks = uniform_layers(model, caches)
        if blocks is None:
            return None
        p = blocks[0].mixer.params
        if p.hidden_size % 8 or blocks[0].ffn.params.intermediate_size % 8:
            return None
        fns = [_library("cublasGemmEx"), _library("cublasSetMathMode")]
        if None in fns:
            return None
        return PromptLayers(model, blocks, caches, ctx, fns)

    def __init__(self, model, blocks, caches, ctx, library):
        rt, ws = model.rt, model.rt.workspace
        att, ffn, norm = blocks[0].mixer, blocks[0].ffn, blocks[0].mixer_norm
        p, self.mixer, self.group, self.rt = att.params, att, caches[0].group, rt
        H, I, T = p.hidden_size, ffn.params.intermediate_size, rt.max_tokens
        attn = kernels._attn(p.head_dim)
        ours = [(kernels._ew(), "rl_add_rmsnorm"), (kernels._ew(), "rl_rope_kv_write"), (attn, "rl_attn_decode"),
                (attn, "rl_attn_prefill"), (kernels._lib("gemm_tc", "gemm_tc.cu"), "rl_gemm_tc"),
                (kernels._lib("gemm_mid", "gemm_mid.cu"), "rl_gemm_mid"), (kernels._ew(), "rl_swiglu")]
        fns = list(library) + [getattr(lib, name) for lib, name in ours]
        counters = [b.mixer._counters(ctx.max_items) for b in blocks]
        self.made_at = Watched.last_change                       # (the counters are kept in an attribute)
        rows = [[b.mixer.w_qkv, b.mixer.w_o, b.ffn.w_gate_up, b.ffn.w_down, b.mixer_norm.weight, b.ffn_norm.weight, c.k, c.v,
                 n] for b, c, n in zip(blocks, caches, counters)]
        self.layers = (_Layer * len(rows))(*[_Layer(*[t.data_ptr() for t in row]) for row in rows])
        bf16, f32, mid = torch.bfloat16, torch.float32, kernels.MID_MAX_ROWS
        tiles = kernels.mid_sum_columns(H)
        # (the buffers that the parts use, by the same names)
        self.residual = ws.get("residual", (T, H), f32)
        self.ffn_out = ws.get("ffn.out", (T, H), bf16)
        buffers = [self.residual, ws.get("block.normed", (T, H), bf16), ws.get("attn.qkv", (T, att.qkv_size), bf16),
                   ws.get("attn.out", (T, att.q_size), bf16), ws.get("mixer.out", (T, H), bf16), ws.get("ffn.act", (T, I), bf16),
                   ws.get("ffn.gate_up", (min(T, TC_MIN_ROWS), 2 * I), bf16), self.ffn_out,
                   ws.get("attn.mid.hand_xw", (mid, H), bf16), ws.get("ffn.mid.hand_xw", (mid, H), bf16),
                   ws.get("attn.mid.hand_sums", (mid, tiles), f32), ws.get("ffn.mid.hand_sums", (mid, tiles), f32)]
        cos, sin = att.position.rotary_tables()
        self.plan = _Plan(*[ctypes.cast(f, c_void_p).value for f in fns], ctypes.addressof(self.layers),
                          *[t.data_ptr() for t in buffers], None, None, cos.data_ptr(), sin.data_ptr(), ctx.status.data_ptr(),
                          kernels.tc_status(rt.device).data_ptr(), caches[0].k.shape[0] * rt.page_size, norm.params.eps, att.scale,
                          len(rows), H, I, p.num_heads, p.num_kv_heads, p.head_dim, rt.page_size, p.window, cos.shape[0],
                          kernels.sm_count(rt.device), TC_MIN_ROWS, tiles)
        self.kept = (rows, buffers, cos, sin, ctx.status)        # what the addresses point at
        self.launch = kernels._fn(kernels._lib("prompt_layers", "prompt_layers.cpp"), "rl_prompt_layers",
                                  [c_void_p, c_void_p, c_int, c_void_p])
        # what ``fits`` compares
        self.spec, self.blocks, self.caches = model.spec, list(model.blocks), list(caches)
        self.weights = [t for row in rows for t in row[:6]]
        self.addresses = list(map(torch.Tensor.data_ptr, self.weights))
        self.sizes = self._sizes(ctx)

    @staticmethod
    def _sizes(ctx) -> tuple:
        return ctx.status.data_ptr(), ctx.max_items, ctx.parts_capacity

    def fits(self, model, caches: List[object], ctx) -> bool:
        """Whether model and step are still what the plan was made for: weights can be loaded again or moved, a part be put
        in another's place, a method be wrapped, and a step can come with other caches or from another batch builder."""
        return (self.made_at == Watched.last_change and self.sizes == self._sizes(ctx) and self.spec is model.spec
                and len(self.blocks) == len(model.blocks) and all(map(is_, self.blocks, model.blocks))
                and len(self.caches) == len(caches) and all(map(is_, self.caches, caches))
                and self.addresses == list(map(torch.Tensor.data_ptr, self.weights)))

    @staticmethod
    def takes(ctx) -> bool:
        """Whether the step goes this way (``REDLINE_PROMPT_LAYERS=0``: never)."""
        return (ctx.T > kernels.SKINNY_MAX_ROWS and ctx.num_tiles > 0 and ctx.profiler is None and not ctx.float32_sums
                and os.environ.get("REDLINE_PROMPT_LAYERS", "1") != "0"
                and (ctx.T > kernels.MID_ROUTED_ROWS or (os.environ.get("REDLINE_MID_PRODUCTS", "1") != "0"
                                                         and os.environ.get("REDLINE_NORM_HANDOVER", "1") != "0")))

    def run(self, ctx) -> Optional[torch.Tensor]:
        """Takes the step's embeddings in the stream's buffer through all layers; returns what is still to be added to the
        stream (None: nothing)."""
        g, few = ctx.groups[self.group], ctx.T <= kernels.MID_ROUTED_ROWS
        if ctx.num_decode > 0 and not self.plan.part_o:
            # (asked for by the first step with single tokens: 2 GB for 256 sequences of up to 131,072 tokens with 32 heads)
            ws, p = self.rt.workspace, self.mixer.params
            n = ctx.max_items * p.num_heads * ctx.parts_capacity
            self.parts = ws.get("attn.part_o", (n * p.head_dim,), torch.float32), ws.get("attn.part_ml", (n * 2,), torch.float32)
            self.plan.part_o, self.plan.part_ml = (t.data_ptr() for t in self.parts)
        step = _Step(0 if few else torch.cuda.current_blas_handle(), kernels._stream(), ctx.positions.data_ptr(),
                     g.slots.data_ptr(), g.block_table.data_ptr(), ctx.decode_info.data_ptr(), ctx.tile_seq.data_ptr(),
                     ctx.tile_tok.data_ptr(), ctx.tile_rows.data_ptr(), ctx.T, g.block_table.shape[1], ctx.num_decode,
                     ctx.decode_parts, ctx.num_tiles, self.mixer.decode_variant(ctx) if ctx.num_decode > 0 else 0)
        n = _Counts()
        code = self.launch(ctypes.addressof(self.plan), ctypes.addressof(step), 1 if few else 0, ctypes.addressof(n))
        if code != 0 and n.failed < 2:
            raise kernels.KernelError(f"{_LAUNCHERS[n.failed]}: cuBLAS status {code}")
        kernels._check(code, _LAUNCHERS[n.failed], n.launches)
        return None if few else self.ffn_out[:ctx.T]
