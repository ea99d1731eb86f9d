"""Decode steps of dense decoders through one resident kernel (csrc/decode_layers.cu).

A model whose every layer is the plain pre-norm decoder layer (RMSNorm, grouped-query attention without biases or head
norms, RMSNorm, SwiGLU) and whose head is a plain matrix can take a step of a few rows, one new token each, in one launch
for all layers and the head, replayed or launched from the host alike (the same bits).  Everything else, and every step this
does not take, runs part by part.
"""
from __future__ import annotations

from typing import NamedTuple, Optional

import torch

from .. import kernels as K
from ..cache.pages import PAGE_TOKENS
from ..parts.attention import GQAAttention
from ..parts.block import PreNormResidual
from ..parts.embedding import LinearHead
from ..parts.linear import Linear
from ..parts.mlp import SwiGLU
from ..parts.norm import RMSNorm
from ..parts.rope import RotaryTable


# Models of fewer layers run part by part: the kernel's set-up (lists of pages, the ring's first filling, the head's tiles) is a
# large share of so short a step.  A step in us, parts / kernel, behind 200 tokens with a vocabulary of 2,048, at one, two and
# four layers: width 512, 8 rows 29 / 33, 47 / 49, 86 / 82; 1 row 36 / 33, 64 / 49, 117 / 82; width 4,096 (8B shape), 8 rows
# 122 / 112, 218 / 194, 409 / 361.
MIN_LAYERS = 4


class Decoder(NamedTuple):
    """A model's parts as the kernel takes them."""
    att: GQAAttention                 # any layer's: the sizes, window, scale and rotation that all have
    rot: Optional[RotaryTable]
    stops: list                       # of every stop of the schedule: (mixer_norm, mixer, feed_forward_norm, feed_forward)


def _is(part, kind) -> bool:
    """Exactly that part, run as it was written (not a subclass, no `forward` of the object's own)."""
    return type(part) is kind and "forward" not in vars(part)


def _copies(t) -> bool:
    """Whether the kernel's 16-byte copies can read it (the parts have kernels for what they cannot)."""
    return t.is_contiguous() and t.data_ptr() % 16 == 0


def _plain(linear) -> bool:
    return type(linear) is Linear and linear.bias is None and _copies(linear.weight)


class ResidentSteps:
    """Which of a model's steps the kernel takes, and how it is called.  Nothing of the model is kept: its parts are looked at
    anew at every step that is not replayed, as the part-by-part path does."""

    refused = False

    @classmethod
    def of(cls, model) -> Optional["ResidentSteps"]:
        """None where the model is not made of the parts the kernel knows, in sizes it takes."""
        return cls() if cls.describe(model) is not None else None

    @staticmethod
    def describe(model) -> Optional[Decoder]:
        rt = model.runtime
        if rt is None or rt.dtype != torch.bfloat16 or rt.device.type != "cuda" or PAGE_TOKENS != 64:
            return None
        if not _is(model.final_norm, RMSNorm) or not _is(model.head, LinearHead) or model.spec.keep_embedded:
            return None
        if any(e.cache_of is not None for e in model.schedule) or not MIN_LAYERS <= len(model.schedule) <= K.DECODE_LAYERS_MAX:
            return None
        eps, shapes, stops = model.final_norm.eps, set(), []
        for e in model.schedule:
            layer = model.layers[e.layer]
            norm_a, att = layer.part("mixer_norm"), layer.part("mixer")
            norm_b, ff = layer.part("feed_forward_norm"), layer.part("feed_forward")
            if not (_is(layer.arrangement, PreNormResidual) and _is(norm_a, RMSNorm) and _is(norm_b, RMSNorm)
                    and _is(att, GQAAttention) and _is(ff, SwiGLU)):
                return None
            if norm_a.eps != eps or norm_b.eps != eps or att.bias or att.q_norm is not None or att.k_norm is not None:
                return None
            if ff.bias or ff.act != K.ACT_NONE or att.hidden != model.hidden:
                return None
            if not (_plain(att.qkv) and _plain(att.o) and _plain(ff.gate_up) and _plain(ff.down)
                    and _copies(norm_a.gain) and _copies(norm_b.gain)):
                return None
            rot = att.position.rotary() if att.position is not None else None
            shapes.add((att.n_heads, att.n_kv_heads, att.head_dim, att.window, att.scale, ff.intermediate,
                        None if rot is None else rot.key))
            stops.append((norm_a, att, norm_b, ff))
        if len(shapes) != 1 or not _plain(model.head.proj) or not _copies(model.final_norm.gain):
            return None
        if not K.decode_layers_sizes_ok(model.hidden, ff.intermediate, model.vocab, att.n_heads, att.n_kv_heads, att.head_dim,
                                        rt.device):
            return None
        return Decoder(att, rot, stops)

    @staticmethod
    def takes(decoder: Decoder, step) -> bool:
        """Whether the kernel takes this step of a model it knows.  Asked of the sizes that a replay of the step has, so that a
        step takes the same way, and gives the same bits, replayed or launched."""
        from .graphs import padded_rows, width_bucket
        rows, width = padded_rows(step.n_tokens), width_bucket(next(iter(step.block_tables.values())).stride(0))
        return K.decode_layers_takes(rows, decoder.att.n_kv_heads, width, step.token_ids.device)

    def run(self, model, x: torch.Tensor, step, cache) -> Optional[torch.Tensor]:
        """Float32 logits of the step's wanted rows; x: the embedded tokens.  None where the step is not one the kernel takes, or
        the launch was refused because not all of its blocks can be resident (`refused` is then set); x is as it was."""
        # (not by whose logits are wanted: what a step leaves in the cache does not depend on that)
        if not (step.all_single and 0 < step.n_tokens <= K.DECODE_LAYERS_MAX_ROWS and step.n_seqs == step.n_tokens
                and len(step.block_tables) == 1):
            return None
        d = self.describe(model)
        if d is None or not self.takes(d, step):
            return None
        m, att = model, d.att
        gains = [stop[0].gain for stop in d.stops] + [m.final_norm.gain]
        layers, table = [], None
        for i, (_, mix, norm_b, ff) in enumerate(d.stops):
            view = cache.layer_view(i, True, step.block_tables)
            table = view.block_table
            layers.append((mix.qkv.weight, mix.o.weight, ff.gate_up.weight, ff.down.weight, norm_b.gain, gains[i + 1],
                           view.k, view.v))
        n_want = step.want_rows.numel()
        logits = torch.empty((step.n_tokens, m.vocab), dtype=torch.float32, device=x.device) if n_want else None
        if not K.decode_layers(x, layers, gains[0], m.head.proj.weight, logits,
                               None if d.rot is None else step.rotation_table(d.rot), step.token_pos, step.token_seq,
                               table, att.n_heads, att.n_kv_heads, att.head_dim, att.window, att.scale, m.final_norm.eps):
            self.refused = True                            # (before anything is captured: a first launch warms up)
            return None
        if logits is None:
            return torch.empty((0, m.vocab), dtype=torch.float32, device=x.device)
        if step.host and step.host.get("want_all"):
            return logits
        return logits.index_select(0, step.want_rows)      # (the head's matrix is read once for all rows anyway)
