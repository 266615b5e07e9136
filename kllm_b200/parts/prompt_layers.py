"""All layers of a prompt's step, launched from one native call (csrc/prompt_layers.cu).

``PromptLayers.of(model)`` is None unless every layer of the model is a pre-norm block of
rotary attention over its own cache and a gated silu feed-forward with plain RMS norms, all
of one size, in bfloat16 (the Llama layer).  ``takes(ctx, caches)`` says whether a step goes
that way: more tokens than the weight-streaming products take, portions among them, a head
size of the tcgen05 attention, and so little work that the host's launches would be the longer
part.  The kernels, their arguments and their order are those of the blocks' own forward;
weights, tables of angles and cache pages are named at every call, and from a layer on where one does not fit the
blocks' own forward runs.
"""
from __future__ import annotations

from .. import kernels
from .attention import PagedAttention
from .block import PreNormBlock
from .mlp import GatedMLP
from .norm import RMSNorm

import torch

# Steps of up to so many operations in a layer's products go this way.  The parts' own launches take 0.16 ms a layer on the
# host; where a layer is less GPU work than that they are the step's time, above it the two are level and the parts run.
# Passes that find the GPU idle, in turn (us, median [quartiles] of 20, this way / parts): TinyLlama's sizes, 300 tokens
# (0.26e11) 2166 [2155 2179] / 3635 [3613 3660], 1200 (1.06e11) 3607 [3594 3633] / 3664 [3639 3705], 1704 (1.5e11) 4949
# [4892 5005] / 4985 [4901 5082] and 4871 [4837 4935] / 4828 [4802 4932], 2048 (1.8e11) 5479 [5436 5518] / 5449
# [5424 5471]; eight Llama-2-7B layers, 24 tokens and 525 of prompts (2.2e11) 3634 [3595 3675] / 3582 [3542 3632].
MOST_WORK = 1.5e11


def _plain_attention(m) -> bool:
    return (type(m) is PagedAttention and not m.window and m.qk_transform is None and m.score_slopes is None
            and m.v_head_dim == m.head_dim and not m.exact_weights and not m.segment and not m.keep_first
            and m.maps == 1 and not m.gate_name and m.out_factor == 1.0 and m.sinks is None and not m.has_bias
            and m.mix_name is None and m.position is not None
            and getattr(m.position, "full_rotary_table", lambda: None)() is not None)


class PromptLayers:
    def __init__(self, model):
        self.blocks = [model.blocks[call.block] for call in model.schedule]
        self.slots = [call.cache for call in model.schedule]
        m, f = self.blocks[0].mixer, self.blocks[0].feed_forward
        self.d, self.heads, self.kv, self.head_dim, self.inter = m.hidden, m.n_heads, m.n_kv, m.head_dim, f.inter
        self.eps, self.scale = self.blocks[0].mixer_norm.eps, m.scale
        self.weights = m.w_qkv.numel() + m.w_o.numel() + f.w_gate_up.numel() + f.w_down.numel()      # of one layer

    @staticmethod
    def of(model):
        if model.dtype != torch.bfloat16 or model.device.type != "cuda" or not model.schedule or model.entries:
            return None
        first = None
        for call in model.schedule:
            b = model.blocks[call.block]
            if type(b) is not PreNormBlock or not call.writes_cache or call.entry is not None:
                return None
            m, f = b.mixer, b.feed_forward
            if not _plain_attention(m) or type(f) is not GatedMLP or not f.plain:
                return None
            if type(b.mixer_norm) is not RMSNorm or type(b.ff_norm) is not RMSNorm:
                return None
            if not all(w.is_contiguous() and w.data_ptr() % 16 == 0 for w in (
                    m.w_qkv, m.w_o, f.w_gate_up, f.w_down, b.mixer_norm.gain, b.ff_norm.gain)):
                return None
            key = (m.hidden, m.n_heads, m.n_kv, m.head_dim, m.scale, f.hidden, f.inter, b.mixer_norm.eps, b.ff_norm.eps)
            if m.hidden != f.hidden or b.mixer_norm.eps != b.ff_norm.eps or (first is not None and key != first):
                return None
            first = first or key
        return PromptLayers(model)

    def takes(self, ctx, caches) -> bool:
        group = self.heads // self.kv
        if 2.0 * ctx.n_tokens * self.weights > MOST_WORK:
            return False
        if (ctx.all_single or not ctx.host_n_new or ctx.n_tokens <= kernels.SKINNY_MAX_ROWS or group > 64
                or not kernels.USE_TCGEN05 or self.head_dim not in kernels.TCGEN05_HEAD_DIMS):
            return False
        c = caches[self.slots[0]]
        return kernels.prompt_layers_ready() and all(
            caches[i].block_table is c.block_table and caches[i].k.shape[2] == c.page_size for i in self.slots)

    def run(self, x, ctx, caches) -> None:
        def operands():
            for b, i in zip(self.blocks, self.slots):
                m, f, c = b.mixer, b.feed_forward, caches[i]
                yield (m.w_qkv, m.w_o, f.w_gate_up, f.w_down, b.mixer_norm.gain, b.ff_norm.gain, c.k, c.v,
                       m.position.full_rotary_table())
        done = kernels.prompt_layers(x, operands(), len(self.blocks), ctx, caches[self.slots[0]].block_table, self.heads, self.kv,
                                     self.head_dim, self.inter, self.eps, self.scale)
        for b, i in zip(self.blocks[done:], self.slots[done:]):      # from an operand that does not fit on: the parts
            b.forward(x, None, ctx, caches[i])
