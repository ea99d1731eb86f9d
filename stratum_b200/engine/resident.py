"""Decode steps of dense decoders through one resident kernel (csrc/decode_layers.cu).

A model whose every layer is the plain pre-norm decoder layer (RMSNorm, grouped-query attention without biases or head
norms, RMSNorm, SwiGLU) and whose head is a plain matrix can take a step of a few rows, one new token each, in one launch
for all layers and the head, replayed or launched from the host alike (the same bits).  Everything else, and every step this
does not take, runs part by part.
"""
from __future__ import annotations

from typing import Optional

import torch

from .. import kernels as K
from ..cache.pages import PAGE_TOKENS
from ..parts.attention import GQAAttention
from ..parts.block import PreNormResidual
from ..parts.embedding import LinearHead
from ..parts.mlp import SwiGLU
from ..parts.norm import RMSNorm


# Models of fewer layers run part by part: the kernel's set-up (lists of pages, the ring's first filling, the head's tiles) is a
# large share of so short a step.  A step in us, parts / kernel, behind 200 tokens with a vocabulary of 2,048, at one, two and
# four layers: width 512, 8 rows 29 / 33, 47 / 49, 86 / 82; 1 row 36 / 33, 64 / 49, 117 / 82; width 4,096 (8B shape), 8 rows
# 122 / 112, 218 / 194, 409 / 361.
MIN_LAYERS = 4


class ResidentSteps:
    """The plan of one model: which of its steps the kernel takes, and how it is called.  (It does not hold the model, which
    holds it: a model's weights go when the last reference to it goes.)"""

    def __init__(self, model):
        self.att = model.layers[model.schedule[0].layer].part("mixer")
        self.rot = self.att.position.rotary() if self.att.position is not None else None

    @classmethod
    def of(cls, model) -> Optional["ResidentSteps"]:
        """The plan, or None where the model is not made of the parts the kernel knows, in sizes it takes."""
        rt = model.runtime
        if rt is None or rt.dtype != torch.bfloat16 or rt.device.type != "cuda" or PAGE_TOKENS != 64:
            return None
        if type(model.final_norm) is not RMSNorm or type(model.head) is not LinearHead or model.spec.keep_embedded:
            return None
        if any(e.cache_of is not None for e in model.schedule) or not MIN_LAYERS <= len(model.schedule) <= K.DECODE_LAYERS_MAX:
            return None
        eps, shapes = model.final_norm.eps, set()
        for e in model.schedule:
            layer = model.layers[e.layer]
            norm_a, att = layer.part("mixer_norm"), layer.part("mixer")
            norm_b, ff = layer.part("feed_forward_norm"), layer.part("feed_forward")
            if (type(layer.arrangement) is not PreNormResidual or type(norm_a) is not RMSNorm or type(norm_b) is not RMSNorm
                    or type(att) is not GQAAttention or type(ff) is not SwiGLU):
                return None
            if norm_a.eps != eps or norm_b.eps != eps or att.bias or att.q_norm is not None or att.k_norm is not None:
                return None
            if ff.bias or ff.act != K.ACT_NONE or att.hidden != model.hidden:
                return None
            rot = att.position.rotary() if att.position is not None else None
            shapes.add((att.n_heads, att.n_kv_heads, att.head_dim, att.window, att.scale, ff.intermediate,
                        None if rot is None else rot.key))
        if len(shapes) != 1:
            return None
        ok = K.decode_layers_sizes_ok(model.hidden, ff.intermediate, model.vocab, att.n_heads, att.n_kv_heads, att.head_dim,
                                      rt.device)
        return cls(model) if ok else None

    def takes(self, step) -> bool:
        # (not by whose logits are wanted: what a step leaves in the cache does not depend on that)
        if not (step.all_single and 0 < step.n_tokens <= K.DECODE_LAYERS_MAX_ROWS and step.n_seqs == step.n_tokens
                and len(step.block_tables) == 1):
            return False
        width = next(iter(step.block_tables.values())).stride(0)
        return K.decode_layers_takes(step.n_tokens, self.att.n_kv_heads, width, step.token_ids.device)

    def run(self, model, x: torch.Tensor, step, cache) -> Optional[torch.Tensor]:
        """Float32 logits of the wanted rows of a step that `takes` accepted; x: the embedded tokens.  None where the launch was
        refused because not all of its blocks can be resident (x is as it was)."""
        m, att = model, self.att
        gains = [m.layers[e.layer].part("mixer_norm").gain for e in m.schedule] + [m.final_norm.gain]
        layers, table = [], None
        for i, e in enumerate(m.schedule):
            layer = m.layers[e.layer]
            mix, ff = layer.part("mixer"), layer.part("feed_forward")
            view = cache.layer_view(i, True, step.block_tables)
            table = view.block_table
            layers.append((mix.qkv.weight, mix.o.weight, ff.gate_up.weight, ff.down.weight,
                           layer.part("feed_forward_norm").gain, gains[i + 1], view.k, view.v))
        n_want = step.want_rows.numel()
        logits = torch.empty((step.n_tokens, m.vocab), dtype=torch.float32, device=x.device) if n_want else None
        if not K.decode_layers(x, layers, gains[0], m.head.proj.weight, logits,
                               None if self.rot is None else step.rotation_table(self.rot), step.token_pos, step.token_seq,
                               table, att.n_heads, att.n_kv_heads, att.head_dim, att.window, att.scale, m.final_norm.eps):
            return None
        if logits is None:
            return torch.empty((0, m.vocab), dtype=torch.float32, device=x.device)
        if step.host and step.host.get("want_all"):
            return logits
        return logits.index_select(0, step.want_rows)      # (the head's matrix is read once for all rows anyway)
