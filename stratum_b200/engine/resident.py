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
# 122 / 112, 218 / 194, 409 / 361: wide models would gain with fewer layers too, but they have more.
MIN_LAYERS = 4
WHOLE_PAGES = 8                       # pages of a (sequence, kv head) pair up to which the kernel leaves it to one block


def pays(rows: int, width: int, n_kv: int, head_dim: int, hidden: int, heads_width: int, blocks: int) -> bool:
    """Whether a step is shorter in the kernel than part by part; `width`: pages it may read of a sequence.  Both were
    measured as replayed steps of 16 layers (us, parts / kernel), 14 shapes behind 200 to 32,000 keys.

    Up to 8 rows, short sequences (no pair is cut): always (Llama-3.2-1B shape, 1 and 8 rows behind 500 keys 862 / 667 and
    934 / 720; 8B 1,713 / 1,494 and 1,754 / 1,563; width 768, 12 layers, 8 rows 322 / 292).
    9 to 16 rows, a second accumulator and twice the rows of x a phase: up to a width of 3,072 (16 rows behind 500: 1B
    989 / 909, 3,072 wide 1,309 / 1,206, but 7B 1,880 / 1,970 and 8B behind 200 1,772 / 1,825), and cut pairs only up to 16
    pages of 8 kv heads or more (behind 1,000: 1B 1,059 / 1,032, four kv heads 927 / 950; behind 8,000: 1B 1,604 / 1,615).
    Up to 8 rows, cut pairs: the block that merges a pair reads its pieces four at a time, behind an atomic (5 to 8 us a layer),
    and what that is taken from must be there.
    * Narrow models have too little to stream in the meantime: width 768, 12 layers, 8 rows behind 2,500 417 / 452; width
      1,024 behind 2,500 605 / 593, behind 8,000 816 / 857; 2,048 wide (1B) 1,261 / 1,128.
    * Few kv heads make many pieces of a pair: up to one a page, and to all blocks over the kv heads.  1 row: one kv head of
      128 behind 1,000 (16 pieces) 1,013 / 685, behind 8,000 (125) 1,122 / 1,849; four kv heads (up to 37) behind 2,500
      856 / 753 and 1,567 / 1,372, behind 8,000, the worst, 875 / 892 and 1,590 / 1,579; eight (18) 928 / 858.
    * Heads of 64 in quarter pages draw less than attention_stream.cu's whole pages: 32 kv heads, 8 rows, 111 pages a block
      (behind 2,500) 1,258 / 1,132, 221 (behind 8,000) 2,087 / 2,124; 8 kv heads, 8 rows behind 32,000 2,185 / 2,209."""
    if rows > 8:
        return max(hidden, heads_width) <= 3072 and width <= (16 if n_kv >= 8 else WHOLE_PAGES)
    if width <= WHOLE_PAGES:
        return True
    if hidden < (1024 if n_kv >= 8 and width <= 64 else 2048) or min(width, blocks // n_kv) > 40:
        return False
    return head_dim != 64 or rows * n_kv * width <= 111 * blocks


class Decoder(NamedTuple):
    """A model's parts as the kernel takes them."""
    att: GQAAttention                 # any layer's: the sizes, window, scale and rotation that all have
    rot: Optional[RotaryTable]
    stops: list                       # of every stop of the schedule: (mixer_norm, mixer, feed_forward_norm, feed_forward)


def _is(part, kind) -> bool:
    """Exactly that part, run as it was written (not a subclass, no `forward` of the object's own)."""
    return type(part) is kind and "forward" not in part.__dict__


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
        head = model.head
        if not _is(model.final_norm, RMSNorm) or not _is(head, LinearHead) or model.spec.keep_embedded:
            return None
        if type(head.proj) is not Linear or head.proj.bias is not None:
            return None
        if any(e.cache_of is not None for e in model.schedule) or not MIN_LAYERS <= len(model.schedule) <= K.DECODE_LAYERS_MAX:
            return None
        eps, hidden, sizes, stops = model.final_norm.eps, model.hidden, None, []
        for e in model.schedule:
            layer = model.layers[e.layer]
            norm_a, att = layer.part("mixer_norm"), layer.part("mixer")
            norm_b, ff = layer.part("feed_forward_norm"), layer.part("feed_forward")
            if not (_is(layer.arrangement, PreNormResidual) and _is(norm_a, RMSNorm) and _is(norm_b, RMSNorm)
                    and _is(att, GQAAttention) and _is(ff, SwiGLU)):
                return None
            if norm_a.eps != eps or norm_b.eps != eps or att.bias or att.q_norm is not None or att.k_norm is not None:
                return None
            if ff.bias or ff.act != K.ACT_NONE or att.hidden != hidden:
                return None
            qkv, o, gate_up, down = att.qkv, att.o, ff.gate_up, ff.down
            if not type(qkv) is type(o) is type(gate_up) is type(down) is Linear:
                return None
            if not qkv.bias is o.bias is gate_up.bias is down.bias is None:
                return None
            rot = att.position.rotary() if att.position is not None else None
            these = (att.n_heads, att.n_kv_heads, att.head_dim, att.window, att.scale, ff.intermediate,
                     None if rot is None else rot.key)
            if sizes is None:
                sizes = these
            elif these != sizes:
                return None
            stops.append((norm_a, att, norm_b, ff))
        if not K.decode_layers_sizes_ok(hidden, ff.intermediate, model.vocab, att.n_heads, att.n_kv_heads, att.head_dim,
                                        rt.device):
            return None
        return Decoder(att, rot, stops)

    @staticmethod
    def takes(decoder: Decoder, step) -> bool:
        """Whether the kernel takes this step of a model it knows.  Asked of the sizes that a replay of the step has, so that a
        step takes the same way, and gives the same bits, replayed or launched."""
        from .graphs import padded_rows, width_bucket
        rows, width = padded_rows(step.n_tokens), width_bucket(next(iter(step.block_tables.values())).stride(0))
        att, device = decoder.att, step.token_ids.device
        seen = min(width, att.window // PAGE_TOKENS + 2) if att.window > 0 else width
        return (K.decode_layers_takes(rows, att.n_kv_heads, width, device)
                and pays(rows, seen, att.n_kv_heads, att.head_dim, att.hidden, att.n_heads * att.head_dim, K.sm_count(device)))

    def run(self, model, x: torch.Tensor, step, cache) -> Optional[torch.Tensor]:
        """Float32 logits of the step's wanted rows; x: the embedded tokens.  None where the step is not one the kernel takes, or
        the launch was refused, because not all of its blocks can be resident or its copies cannot read a weight (`refused` is then
        set); x is as it was."""
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
