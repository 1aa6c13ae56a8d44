"""Prompt steps and small decode steps of dense models, launched from native code (``csrc/dense_step.cu``, ``csrc/dense_decode.cu``).

A prompt step runs some seven kernels per layer; launched one by one through
the parts they cost the host about 12 us each (2.4 ms per step at 28 layers,
whatever the prompt's length).  Where every layer is the dense decoder's -
pre-norm block, RMS norms, grouped-query attention, SiLU-gated feed-forward,
nothing between the layers - the same launches are made by ``fd_dense_layers``
(up to 128 tokens: the whole step in one call) or, layer by layer, by
``fd_dense_mixer`` and ``fd_dense_gate_up`` around the library products of the
output and down projections.  A decode step of up to 24 sequences is one kernel
for all layers (``fd_dense_decode``) where it takes the sizes.  Everything else, and every step that this module
does not take, goes through the parts' ``forward``.

A part whose ``forward`` was wrapped or replaced, on the object or on its class,
is called: such a model's steps go through the parts.

Kept from step to step: the weights (their memory, too), and their addresses.
A step first looks whether a part has changed since (``Part.changes``) and
derives everything anew if so.  Whether the weights' tensors have been given
other memory takes 10 us to see at 28 layers, so that is asked behind the
launches (``moved``), and such a step runs again through the parts.  The
cache's, the step's and the workspace's addresses are taken anew for every step.
"""

from __future__ import annotations

import ctypes
from ctypes import c_double, c_longlong, c_void_p
from typing import List, Optional

import torch

from .. import kernels as K
from ..parts import linear
from ..parts.attention import GQAAttention, prompt_scratch
from ..parts.base import Part
from ..parts.block import PreNormBlock
from ..parts.mlp import SwiGLU
from ..parts.norm import RMSNorm

MAX_GROUPS, MAX_POSITIONS = 8, 4
DECODE_MAX_ROWS = 24         # sequences of a decode step that one kernel takes
KINDS = (PreNormBlock, RMSNorm, GQAAttention, SwiGLU)
FORWARDS = [kind.forward for kind in KINDS]                         # what the native calls stand for
_address = torch.Tensor.data_ptr


class _Layer(ctypes.Structure):
    _fields_ = ([(n, c_void_p) for n in ("norm1", "norm2", "w_qkv", "b_qkv", "w_o", "w_gate_up", "w_down")]
                + [(n, c_longlong) for n in ("norm1_f32", "norm2_f32", "bias_f32", "hidden", "inter", "n_q", "n_kv", "d", "window",
                                             "chunk", "write_kv", "group", "index", "position")]
                + [(n, c_double) for n in ("eps1", "eps2", "scale")])


class _Step(ctypes.Structure):
    _fields_ = ([(n, c_void_p) for n in ("resid", "normed", "q", "attn", "mixer_out", "act", "ffn_out", "tok_row", "tok_pos",
                                         "row_slot", "row_q_start", "row_q_len", "row_ctx_len", "status", "stream",
                                         "attn_scratch")]
                + [(n, c_longlong) for n in ("T", "n_rows", "max_q_len", "kv_len", "num_blocks", "block_size", "streams")]
                + [(n, c_void_p * MAX_GROUPS) for n in ("k_base", "v_base", "table")]
                + [(n, c_longlong * MAX_GROUPS) for n in ("k_stride", "v_stride", "max_blocks")]
                + [(n, c_void_p * MAX_POSITIONS) for n in ("cos", "sin")] + [("table_len", c_longlong * MAX_POSITIONS)])


class _Decode(ctypes.Structure):
    _fields_ = ([(n, c_void_p) for n in ("resid", "tok_pos", "row_slot", "row_ctx_len", "status", "stream", "exchange")]
                + [(n, c_longlong) for n in ("M", "num_blocks", "block_size")]
                + [(n, c_void_p * MAX_GROUPS) for n in ("k_base", "v_base", "table")]
                + [(n, c_longlong * MAX_GROUPS) for n in ("k_stride", "v_stride", "max_blocks")]
                + [(n, c_void_p * MAX_POSITIONS) for n in ("cos", "sin")] + [("table_len", c_longlong * MAX_POSITIONS)]
                + [("next", c_void_p), ("next_bytes", c_longlong)])


class DensePrompts:
    """The native form of a bound model's prompt steps and small decode steps; ``DensePrompts.of(model)`` is None for a
    model that is not of that kind."""

    @staticmethod
    def of(model) -> Optional["DensePrompts"]:
        native = DensePrompts()
        native._derive(model)
        return native if native.layers is not None else None

    def __init__(self):
        # (no reference to the model, which holds this object: a dropped model's weights go at once)
        self.derived_at, self.blocks, self.schedule, self.layers = -1, [], None, None
        self.tensors, self.where, self.memory = [], [], []

    def __reduce__(self):
        """A copied model's is derived from its own parts, at its first step."""
        return DensePrompts, ()

    def _derive(self, model) -> None:
        """The launches' constants from the model's parts as they are now; ``layers`` None: not a model of this kind."""
        self.derived_at = Part.changes                              # before anything is read
        self.blocks, self.schedule = list(model.blocks), model.schedule
        self.tensors, self.where, self.memory = [], [], []
        self.layers = self._layers(model)

    def _layers(self, model):
        if model.dtype != torch.bfloat16 or model.blueprint.lanes != 1 or model.stream_ops:
            return None
        blocks = [self.blocks[run.layer] for run in model.schedule]
        for run, b in zip(model.schedule, blocks):
            if run.before is not None or type(b) is not PreNormBlock or b.side is not None:
                return None
            if type(b.norm1) is not RMSNorm or type(b.norm2) is not RMSNorm or type(b.mixer) is not GQAAttention or \
                    type(b.feed_forward) is not SwiGLU or not (b.mixer.paired and b.feed_forward.tiled):
                return None
            if b.norm1.delta_scale != 1.0 or b.norm2.delta_scale != 1.0 or b.norm1.weight is None or b.norm2.weight is None:
                return None
            if any("forward" in vars(p) for p in (b, b.norm1, b.norm2, b.mixer, b.feed_forward)):
                return None
        sizes = {(b.mixer.n_q, b.mixer.n_kv, b.mixer.d, b.feed_forward.inter) for b in blocks}
        positions = list({id(b.mixer.position): b.mixer.position for b in blocks}.values())
        if len(sizes) != 1 or len(positions) > MAX_POSITIONS or len(model.cache_groups()) > MAX_GROUPS:
            return None
        tensors = [t for b in blocks for t in (b.norm1.weight, b.norm2.weight, b.mixer.w_qkv, b.mixer.b_qkv, b.mixer.w_o,
                                               b.feed_forward.w_gate_up, b.feed_forward.w_down) if t is not None]
        if not blocks or not all(t.is_cuda and t.is_contiguous() for t in tensors):
            return None
        H = model.hidden_size
        for b in blocks:                                            # (replaced weights may be anything)
            m, f = b.mixer, b.feed_forward
            shapes = ((m.w_qkv, ((m.n_q + 2 * m.n_kv) * m.d, H)), (m.w_o, (H, m.n_q * m.d)), (f.w_gate_up, (2 * f.inter, H)),
                      (f.w_down, (H, f.inter)))
            vectors = [(b.norm1.weight, H), (b.norm2.weight, H)] + ([] if m.b_qkv is None else [(m.b_qkv, m.w_qkv.shape[0])])
            if any(w.dtype != torch.bfloat16 or w.shape != shape for w, shape in shapes) or \
                    any(v.dtype not in (torch.bfloat16, torch.float32) or v.shape != (n,) for v, n in vectors):
                return None
        self.tensors, self.where, self.memory = tensors, list(map(_address, tensors)), [t.detach() for t in tensors]
        self.positions, self.n = positions, len(blocks)
        self.hidden = H
        m, f = blocks[0].mixer, blocks[0].feed_forward
        self.n_q, self.n_kv, self.d, self.inter = m.n_q, m.n_kv, m.d, f.inter
        self.qkv = (m.n_q + 2 * m.n_kv) * m.d
        layers = (_Layer * self.n)()
        self.products = []                                          # (w_o^T, w_down^T): the library products' operands
        for i, (b, (gi, li, writes, _)) in enumerate(zip(blocks, model._layout[2])):
            m, f, L = b.mixer, b.feed_forward, layers[i]
            L.norm1, L.norm2 = b.norm1.weight.data_ptr(), b.norm2.weight.data_ptr()
            L.w_qkv, L.b_qkv = m.w_qkv.data_ptr(), None if m.b_qkv is None else m.b_qkv.data_ptr()
            L.w_o, L.w_gate_up, L.w_down = m.w_o.data_ptr(), f.w_gate_up.data_ptr(), f.w_down.data_ptr()
            L.norm1_f32, L.norm2_f32 = b.norm1.weight.dtype == torch.float32, b.norm2.weight.dtype == torch.float32
            L.bias_f32 = m.b_qkv is not None and m.b_qkv.dtype == torch.float32
            L.hidden, L.inter, L.n_q, L.n_kv, L.d = self.hidden, f.inter, m.n_q, m.n_kv, m.d
            L.window, L.chunk, L.write_kv = m.window or 0, m.chunk or 0, int(writes)
            L.group, L.index, L.position = gi, li, [p is m.position for p in positions].index(True)
            L.eps1, L.eps2, L.scale = b.norm1.eps, b.norm2.eps, m.scale
            self.products.append((m.w_o.t(), f.w_down.t()))
        self.addresses = [ctypes.addressof(layers[i]) for i in range(self.n)]
        self.exchange_words = {}                                    # of a decode step, by its rows; 0: not taken
        self.all_write = all(writes for _, _, writes, _ in model._layout[2])
        return layers

    def _current(self, model) -> bool:
        """Whether the model is of the kind, as its parts are now."""
        if self.derived_at != Part.changes or self.blocks != model.blocks or self.schedule is not model.schedule:
            self._derive(model)
        return self.layers is not None and [kind.forward for kind in KINDS] == FORWARDS

    def takes(self, model, ctx) -> bool:
        """Whether the parts would run this step on the kernels that the native calls launch."""
        T = ctx.T
        if linear.PROMPT_GEMM != "auto" or ctx.max_q_len < 2 or T <= linear.GEMV_MAX_ROWS:
            return False
        if not self._current(model):
            return False
        H = self.hidden
        if T <= linear.STREAM_MAX_ROWS:
            return all(linear.stream_gemm(T, n, k) for n, k in ((self.qkv, H), (H, self.n_q * self.d), (2 * self.inter, H), (H, self.inter)))
        return linear.fused_prompt_gemm(T, self.qkv, H) and linear.fused_prompt_gemm(T, 2 * self.inter, H)

    def decodes(self, model, ctx) -> bool:
        """Whether the step is one token each of so few sequences that one kernel runs all of its layers
        (``csrc/dense_decode.cu``); every layer has to write the keys that it reads."""
        T = ctx.T
        if ctx.max_q_len != 1 or T > (DECODE_MAX_ROWS if linear.PROMPT_GEMM == "auto" else linear.GEMV_MAX_ROWS) or T != ctx.n_rows:
            return False
        if not self._current(model) or not self.all_write:
            return False
        if any(g.table.shape[1] * ctx.cache.block_size ** 2 >= 1 << 32 for g in ctx.cache.groups):
            return False                                            # (the kernel divides positions by the block size in 32 bits)
        words = self.exchange_words.get(T)
        if words is None:
            words = self.exchange_words[T] = K.dense_decode_words(T, self.hidden, self.inter, self.n_q, self.n_kv, self.d)
        return words > 0

    def decode(self, ctx, resid: torch.Tensor, upcoming: Optional[torch.Tensor]) -> None:
        """Every schedule entry of the step; ``resid`` is the finished stream then.  ``upcoming``: what the step streams next."""
        s, cache = _Decode(), ctx.cache
        s.resid, s.tok_pos, s.row_slot = resid.data_ptr(), ctx.tok_pos.data_ptr(), ctx.row_slot.data_ptr()
        s.row_ctx_len, s.status, s.stream = ctx.row_ctx_len.data_ptr(), ctx.rt.status.data_ptr(), K._stream()
        # zeroed when it is made; steps of all row counts share it
        s.exchange = ctx.ws.get("dense_decode", (self.exchange_words[ctx.T],), torch.int64).data_ptr()
        s.M = ctx.T
        s.next, s.next_bytes = K._prefetch_args(upcoming, linear.UPCOMING_BYTES)       # (a hint: the head may be any part)
        self._cache_args(s, cache)
        K._check(K.lib().fd_dense_decode(ctypes.addressof(s), self.addresses[0], self.n))

    def _cache_args(self, s, cache) -> None:
        """The pools, tables and rotation tables of a step."""
        s.num_blocks, s.block_size = cache.num_blocks, cache.block_size
        for i, g in enumerate(cache.groups):
            s.k_base[i], s.v_base[i], s.table[i] = g.keys.data_ptr(), g.values.data_ptr(), g.table.data_ptr()
            s.k_stride[i], s.v_stride[i] = 2 * g.keys.stride(0), 2 * g.values.stride(0)
            s.max_blocks[i] = g.table.shape[1]
        for i, p in enumerate(self.positions):
            s.cos[i], s.sin[i], s.table_len[i] = p.cos.data_ptr(), p.sin.data_ptr(), p.cos.shape[0]

    def moved(self, model) -> bool:
        """Whether a weight's tensor has other memory than the step that was just launched used; then everything is derived anew."""
        if list(map(_address, self.tensors)) == self.where:
            return False
        self._derive(model)
        return True

    def run(self, ctx, resid: torch.Tensor) -> torch.Tensor:
        """Every schedule entry of the step; returns the last one's output, still to be added to ``resid``."""
        T, H, ws, cache = ctx.T, self.hidden, ctx.ws, ctx.cache
        bf16 = torch.bfloat16
        normed, q = ws.get("normed", (T, H), bf16), ws.get("q_rot", (T, self.n_q * self.d), bf16)
        attn, mixed = ws.get("attn", (T, self.n_q * self.d), bf16), ws.get("mixer_out", (T, H), bf16)
        act, out = ws.get("ffn_act", (T, self.inter), bf16), ws.get("ffn_out", (T, H), bf16)
        s = _Step()
        s.resid, s.normed, s.q, s.attn = resid.data_ptr(), normed.data_ptr(), q.data_ptr(), attn.data_ptr()
        s.mixer_out, s.act, s.ffn_out = mixed.data_ptr(), act.data_ptr(), out.data_ptr()
        s.tok_row, s.tok_pos, s.row_slot = ctx.tok_row.data_ptr(), ctx.tok_pos.data_ptr(), ctx.row_slot.data_ptr()
        s.row_q_start, s.row_q_len = ctx.row_q_start.data_ptr(), ctx.row_q_len.data_ptr()
        s.row_ctx_len, s.status, s.stream = ctx.row_ctx_len.data_ptr(), ctx.rt.status.data_ptr(), K._stream()
        s.T, s.n_rows, s.max_q_len, s.kv_len = T, ctx.n_rows, ctx.max_q_len, ctx.kv_len_bound
        scratch = prompt_scratch(ctx, self.n_q, self.d)
        s.attn_scratch = None if scratch is None else scratch.data_ptr()
        s.streams = T <= linear.STREAM_MAX_ROWS
        self._cache_args(s, cache)
        L, step = K.lib(), ctypes.addressof(s)
        if s.streams:
            K._check(L.fd_dense_layers(step, self.addresses[0], self.n))
            return out
        delta = None
        for address, (w_o, w_down) in zip(self.addresses, self.products):
            K._check(L.fd_dense_mixer(step, address, delta))
            torch.mm(attn, w_o, out=mixed)
            K._check(L.fd_dense_gate_up(step, address))
            torch.mm(act, w_down, out=out)
            delta = s.ffn_out
        return out
