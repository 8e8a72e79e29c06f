"""The composite Pairformer block the benchmark configurations describe, and its stack.

Pair track: triangle multiplication outgoing / incoming, triangle attention starting / ending node, pair
transition; single track: attention with pair bias (bias projected from z) and a transition; every
sub-block is residual.  The reference's own trunk block (``PairMixerLayer``, ``bioemu2_b200.pairmixer``) is
the first two and the fifth of these (src/bioemu2/biomoa/modules/pairmixer.py:430-456); the attention
sub-blocks are ``AttentionPairBias`` (src/bioemu2/biomoa/ops/attention_pair_bias.py:42) and the triangle
attention of ``bioemu2_b200.triangle_attention``, which the reference lacks.

Sub-module names: ``tri_mul_out``, ``tri_mul_in``, ``tri_att_start``, ``tri_att_end``, ``transition_z``,
``attention``, ``transition_s``.
"""
from __future__ import annotations

import torch
import torch.nn as nn
from torch import Tensor

from . import _lib, precision
from . import functional as F
from .attention_pair_bias import AttentionPairBias
from .transition import Transition
from .triangle_attention import TriangleAttention, TriangleAttentionEndingNode, TriangleAttentionStartingNode
from .triangle_multiplication import PackedWeightsMixin, TriangleMultiplication, native_trimul


_OWN_TRIATT = (TriangleAttention, TriangleAttentionStartingNode, TriangleAttentionEndingNode)


class PairformerBlock(nn.Module):
    def __init__(self, token_s: int = 384, token_z: int = 128, tri_heads: int = 4, tri_head_dim: int = 32,
                 apb_heads: int = 16) -> None:
        super().__init__()
        self.tri_mul_out = TriangleMultiplication(token_z, "outgoing")
        self.tri_mul_in = TriangleMultiplication(token_z, "incoming")
        self.tri_att_start = TriangleAttention(token_z, tri_heads, tri_head_dim, ending=False)
        self.tri_att_end = TriangleAttention(token_z, tri_heads, tri_head_dim, ending=True)
        self.transition_z = Transition(token_z, 4 * token_z)
        self.attention = AttentionPairBias(token_s, token_z, apb_heads)
        self.transition_s = Transition(token_s, 4 * token_s)

    def forward_(self, s: Tensor, z: Tensor, token_mask: Tensor, pair_mask_u8: Tensor) -> tuple[Tensor, Tensor]:
        """In-place form: updates ``s`` and ``z`` (contiguous, fp32 or bf16) and returns them."""
        self.tri_mul_out.forward_residual_(z, pair_mask_u8)
        self.tri_mul_in.forward_residual_(z, pair_mask_u8)
        self.tri_att_start.forward_residual_(z, pair_mask_u8)
        self.tri_att_end.forward_residual_(z, pair_mask_u8)
        self.transition_z.forward_residual_(z)
        s += self.attention(s, z, token_mask)
        self.transition_s.forward_residual_(s)
        return s, z

    def forward(self, s: Tensor, z: Tensor, token_mask: Tensor) -> tuple[Tensor, Tensor]:
        if self.training:
            raise RuntimeError("bioemu2_b200 modules are inference-only: call .eval()")
        pm = (token_mask[:, :, None] & token_mask[:, None, :]).to(torch.uint8)
        return self.forward_(s.clone(), z.clone(), token_mask, pm)


class PairformerModule(PackedWeightsMixin, nn.Module):
    def __init__(self, token_s: int = 384, token_z: int = 128, num_blocks: int = 48, **block_kwargs) -> None:
        super().__init__()
        self.num_blocks = num_blocks
        self.layers = nn.ModuleList([PairformerBlock(token_s, token_z, **block_kwargs) for _ in range(num_blocks)])

    @staticmethod
    def _native(m) -> bool:
        """Whether the native call covers a block: one with a module or a path of its own runs by itself."""
        if type(m) is not PairformerBlock:
            return False
        op = m._modules  # (looked up on every pass, and a module's own getattr is ten times a dict's)
        start, end, tz, attention, ts = (op[k] for k in ("tri_att_start", "tri_att_end", "transition_z", "attention", "transition_s"))
        return native_trimul(op["tri_mul_out"], "outgoing") and native_trimul(op["tri_mul_in"], "incoming") \
            and type(start) in _OWN_TRIATT and not start.ending and type(end) in _OWN_TRIATT and end.ending \
            and type(tz) is Transition and tz._fused and type(attention) is AttentionPairBias and attention._bias_cache is None \
            and type(ts) is Transition and not ts._fused

    def _pack_block(self, i: int) -> dict:
        m = self.layers[i]
        return {"tri_mul_out": m.tri_mul_out.packed(), "tri_mul_in": m.tri_mul_in.packed(),
                "tri_att_start": m.tri_att_start.packed(), "tri_att_end": m.tri_att_end.packed(),
                "transition_z": m.transition_z.packed(), "attention": m.attention.packed(),
                "transition_s": m.transition_s.packed()}

    def forward(self, s: Tensor, z: Tensor, token_mask: Tensor) -> tuple[Tensor, Tensor]:
        if self.training:
            raise RuntimeError("bioemu2_b200 modules are inference-only: call .eval()")
        s = s.clone(memory_format=torch.contiguous_format)
        z = self.forward_into(s, F.aligned(z.contiguous()), torch.empty_like(z, memory_format=torch.contiguous_format), token_mask)
        _lib.raise_if_device_wait()  # a kernel whose bounded wait ran out earlier in the stack invalidates the result
        return s, z

    def forward_(self, s: Tensor, z: Tensor, token_mask: Tensor, pair_mask_u8: Tensor | None = None, overlap: bool = True):
        """The block loop in place on contiguous ``s`` and ``z``; ``pair_mask_u8=None``: the outer product of the token mask."""
        self.forward_into(s, z, z, token_mask, pair_mask_u8, overlap)
        return s, z

    def forward_into(self, s: Tensor, z_in: Tensor, z: Tensor, token_mask: Tensor, pair_mask_u8: Tensor | None = None,
                     overlap: bool = True) -> Tensor:
        """The block loop: ``s`` in place, ``z_in`` -> ``z`` (contiguous; ``z`` may be ``z_in``); returns ``z``.

        The whole stack is one native call (``b200_trunk_fwd``).  The pair track never reads the single track, and the
        single track needs from the pair track only the 16-head attention bias of the block's final ``z``.  With
        ``overlap`` that bias is projected on the current stream right after the block's pair transition, and the rest of
        the block's single track - a handful of small, launch-bound kernels - runs on a side stream underneath the pair
        track of the NEXT block; the streams join at the end of the stack.  Both forms launch the same kernels on the same
        data and give identical results.
        """
        native = len(self.layers) > 0 and not precision.use_ieee(None, s, z) and all(self._native(m) for m in self.layers)
        if not native:  # a layer with a module or a path of its own (accurate mode, adopted bias cache, 128-wide single track)
            if z is not z_in:
                z.copy_(z_in)
            if pair_mask_u8 is None:
                pair_mask_u8 = (token_mask[:, :, None] & token_mask[:, None, :]).to(torch.uint8)
            for layer in self.layers:
                layer.forward_(s, z, token_mask, pair_mask_u8)
            return z
        side = None
        if overlap:
            if self._side is None or self._side.device != z.device:
                self._side = torch.cuda.Stream(device=z.device)
            side = self._side
        heads = self.layers[0].attention.num_heads
        done = False

        def first_run():
            nonlocal done
            done = True
            return F.trunk_blocks_(z_in, z, s, token_mask, pair_mask_u8, self._pack_block, len(self.layers), heads, side)

        w = self.packed(first_run)
        if not done:
            F.trunk_(z_in, z, s, token_mask, pair_mask_u8, w, heads, side)
        return z

    _side = None

    def graphed(self, s: Tensor, z: Tensor, token_mask: Tensor):
        """The block loop captured in a CUDA graph for inputs of these shapes: ``g = trunk.graphed(s, z, mask)`` once,
        then ``s_out, z_out = g(s, z[, mask])`` per forward (see ``bioemu2_b200.graph``)."""
        from .graph import GraphedTrunk

        return GraphedTrunk(self, s, z, token_mask)
