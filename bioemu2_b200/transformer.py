"""Token block of the diffusion module: ``ConditionedTransformerLayer`` with full attention
(src/bioemu2/biomoa/modules/transformer.py:231-353, ``ada_ln`` :26-41, ``AttentionLayer`` :54-135).

    alpha1, beta1, gamma1, alpha2, beta2, gamma2 = cond(c).chunk(6)        cond = LayerNorm -> SiLU -> Linear
    x += gamma1 * APB(lns * ((1 + alpha1) * LN(x) + beta1), pairs, mask)
    x += gamma2 * Transition(lns * ((1 + alpha2) * LN(x) + beta2))         Transition without its own norm

Same sub-module names as the reference (``cond.0``, ``cond.2``, ``attention.pair_bias_attn``, ``transition``),
so its state_dict loads unchanged.  With ``is_sliding_window=True`` the attention is the atom transformer's windowed
one (``SlidingWindowAttentionLayer`` :147-229 around ``AttentionPairBiasSlidingWindow``): same block, atoms in place of
tokens, the pair tensor pre-windowed ``[B, NW, W, H, dim_pairwise]``.
"""
from __future__ import annotations

import torch
import torch.nn as nn
from torch import Tensor

from . import _lib
from . import functional as F
from .attention_pair_bias import AttentionPairBias, AttentionPairBiasSlidingWindow
from .transition import Transition
from .triangle_multiplication import PackedWeightsMixin, plain


class AttentionLayer(nn.Module):
    def __init__(self, heads: int, dim: int = 384, dim_pairwise: int = 128,
                 attn_pair_bias_tile_size: int | None = None, is_sliding_window: bool = False,
                 window_queries: int | None = None, window_keys: int | None = None,
                 zero_init_output: bool = False) -> None:
        super().__init__()
        if is_sliding_window:
            assert window_queries is not None and window_keys is not None, (
                "sliding-window AttentionLayer requires window_queries / window_keys.")
            self.pair_bias_attn = AttentionPairBiasSlidingWindow(
                c_s=dim, c_z=dim_pairwise, num_heads=heads, window_queries=window_queries, window_keys=window_keys,
                initial_norm=False, zero_init_output=zero_init_output)
        else:
            self.pair_bias_attn = AttentionPairBias(
                c_s=dim, c_z=dim_pairwise, num_heads=heads, initial_norm=False, zero_init_output=zero_init_output,
                tile_size=512 if attn_pair_bias_tile_size is None else attn_pair_bias_tile_size)

    def forward(self, tokens: Tensor, pairs: Tensor, mask: Tensor | None = None, multiplicity: int = 1) -> Tensor:
        return self.pair_bias_attn(tokens, pairs, mask, multiplicity)


class SlidingWindowAttentionLayer(nn.Module):
    """Folds atoms into query windows around a windowed ``AttentionLayer`` (transformer.py:147-229):
    ``tokens[B*M, N, dim]``, ``pairs[B, NW, W, H, dim_pairwise]`` (or flat ``[B, N, H, dim_pairwise]``), ``mask[B, N]``."""

    def __init__(self, attn_window_queries: int, attn_window_keys: int, **atom_attention_kwargs) -> None:
        super().__init__()
        assert attn_window_queries > 1 and attn_window_keys > 1
        self.attn_window_queries, self.attn_window_keys = attn_window_queries, attn_window_keys
        self.attention_layer = AttentionLayer(**atom_attention_kwargs, is_sliding_window=True,
                                              window_queries=attn_window_queries, window_keys=attn_window_keys)

    def forward(self, tokens: Tensor, pairs: Tensor, mask: Tensor | None = None, multiplicity: int = 1) -> Tensor:
        W, H = self.attn_window_queries, self.attn_window_keys
        BM, N, D = tokens.shape
        if N % W:
            raise ValueError(f"the atom count {N} is not a multiple of the query window {W}")
        NW = N // W
        B = pairs.shape[0]
        if mask is None:
            mask = torch.ones(B, N, dtype=torch.bool, device=tokens.device)
        out = self.attention_layer(tokens.reshape(BM * NW, W, D), pairs.reshape(B, NW, W, H, -1), mask.reshape(B * NW, W),
                                   multiplicity)
        return out.view(BM, N, D)


class ConditionedTransformerLayer(PackedWeightsMixin, nn.Module):
    def __init__(self, dim: int, dim_pairwise: int, dim_cond: int, heads: int, transition_hidden: int,
                 is_sliding_window: bool = False, window_queries: int | None = None, window_keys: int | None = None,
                 attn_pair_bias_tile_size: int | None = None, lns_scale: float = 1.0) -> None:
        super().__init__()
        self.lns_scale = lns_scale
        self.dim = dim
        self._windowed = is_sliding_window
        self.cond = nn.Sequential(nn.LayerNorm(dim_cond), nn.SiLU(), nn.Linear(dim_cond, 6 * dim))
        if is_sliding_window:
            assert window_queries is not None and window_keys is not None, (
                "sliding-window ConditionedTransformerLayer requires window_queries / window_keys.")
            self.attention: nn.Module = SlidingWindowAttentionLayer(
                attn_window_queries=window_queries, attn_window_keys=window_keys, heads=heads, dim=dim,
                dim_pairwise=dim_pairwise, attn_pair_bias_tile_size=attn_pair_bias_tile_size)
        else:
            self.attention = AttentionLayer(heads=heads, dim=dim, dim_pairwise=dim_pairwise,
                                            attn_pair_bias_tile_size=attn_pair_bias_tile_size)
        self.transition = Transition(dim=dim, hidden=transition_hidden, use_norm=False)

    def _build_packed(self):
        """The conditioning projection in kernel layout, and the native layer's weights where the layer fits it."""
        lin, ln = self.cond[2], self.cond[0]
        pk = F._Pack()
        pk.add(lin.weight)
        w_cond = pk.build(lin.weight.device).view(lin.weight.shape)
        b_cond = lin.bias.detach().float().contiguous()
        ln_w, ln_b = (None if p is None else p.detach().float().contiguous() for p in (ln.weight, ln.bias))
        attn, tr = self._native_attention(lambda m, cls: type(m) is cls), self.transition  # hooks may go again
        native = None
        if attn is not None and self.dim % 32 == 0 and lin.in_features % 8 == 0 and lin.in_features <= 1024 \
                and not tr.use_norm and not attn.initial_norm and ln.eps == 1e-5 and tr.fc3.out_features == self.dim and (self._windowed or attn.c_z == 128):
            layer = _lib.CondLayer()
            ap, tp = attn.packed(), tr.packed()
            layer.dim, layer.dim_cond, layer.heads, layer.dim_pairwise = self.dim, lin.in_features, attn.num_heads, attn.c_z
            layer.ln_c_w, layer.ln_c_b, layer.w_cond, layer.b_cond = F._ptr(ln_w), F._ptr(ln_b), w_cond.data_ptr(), b_cond.data_ptr()
            if self._windowed:
                layer.window_queries, layer.window_keys = attn.window_queries, attn.window_keys
                layer.w_qkvg, layer.b_qkvg, layer.w_o = ap.w_qkvg.data_ptr(), ap.b_qkvg.data_ptr(), ap.w_o.data_ptr()
                layer.ln_z_w, layer.ln_z_b, layer.w_z = ap.ln_z_w.data_ptr(), F._ptr(ap.ln_z_b), ap.w_z.data_ptr()
            else:
                layer.attention = ap.struct
            if tr._fused:
                layer.transition_fused = tp.struct
            else:
                layer.transition = tp.struct
            native = (layer, (ap, tp, ln_w, ln_b))
        return w_cond, b_cond, native

    def _native_attention(self, fits=plain):
        """The attention module whose weights the native call takes, if it may stand for the sub-modules as they are now."""
        attn, own = self._modules["attention"], AttentionPairBias  # (on every pass: a module's own getattr is ten times a dict's)
        if self._windowed:
            if not fits(attn, SlidingWindowAttentionLayer):
                return None
            attn, own = attn._modules["attention_layer"], AttentionPairBiasSlidingWindow
        if not fits(attn, AttentionLayer):
            return None
        attn = attn._modules["pair_bias_attn"]
        return attn if fits(attn, own) and fits(self._modules["transition"], Transition) else None

    def forward(self, x: Tensor, pairs: Tensor, c: Tensor, mask: Tensor | None = None, multiplicity: int = 1) -> Tensor:
        if mask is None:  # full attention: pairs [B, T, T, .]; windowed: x [B*M, atoms, .]
            n = x.shape[1] if pairs.ndim == 5 else pairs.shape[1]
            mask = torch.ones(pairs.shape[0], n, dtype=torch.bool, device=x.device)
        native, attn = self.packed()[2], self._native_attention()
        if native is None or attn is None:
            return self._forward(x, pairs, c, mask, multiplicity, self.attention)
        layer, B, shape, mshape = native[0], pairs.shape[0], x.shape, mask.shape
        N = shape[1] if len(shape) == 3 else -1
        if self._windowed and mshape != (B, N) and mask.numel() == B * N:
            mask = mask.reshape(B, N)  # it may come by query windows
            mshape = mask.shape
        if N < 0 or shape[0] != B * multiplicity or shape[2] != self.dim or mshape != (B, N) \
                or c.shape[-1] != layer.dim_cond or c.numel() != shape[0] * N * layer.dim_cond:
            raise ValueError(f"x {tuple(shape)}, c {tuple(c.shape)}, pairs {tuple(pairs.shape)}, mask {tuple(mshape)}, "
                             f"multiplicity={multiplicity}")
        bias = None
        if self._windowed:
            W, Hk = layer.window_queries, layer.window_keys
            if N % W:
                raise ValueError(f"the atom count {N} is not a multiple of the query window {W}")
            if pairs.numel() != B * N * Hk * layer.dim_pairwise:
                raise ValueError(f"pairs {tuple(pairs.shape)} do not hold {N // W} windows of {W} x {Hk}")
        else:
            if tuple(pairs.shape) != (B, N, N, 128):
                raise ValueError(f"expected pairs[{B},{N},{N},128], got {tuple(pairs.shape)}")
            if attn._bias_cache is not None:
                bias = attn._bias_cache[0].lookup(attn._bias_cache[1], pairs)
        sized = _lib.CondLayer.from_buffer_copy(layer)  # the layer's own copy may be in use by another thread
        sized.B, sized.M, sized.N, sized.lns_scale = B, multiplicity, N, self.lns_scale
        return F.cond_layer(sized, x, pairs, bias, c, mask)

    def _forward(self, x: Tensor, pairs: Tensor, c: Tensor, mask: Tensor, multiplicity: int, attention) -> Tensor:
        """The block with the attention supplied by the caller (``attention(tokens, pairs, mask, multiplicity)``), for the
        context-parallel wrapper's sharded attention and for widths the native layer does not take; everything else is per
        token."""
        w_cond, b_cond, _ = self.packed()
        D = self.dim
        cn = F.rows_to_bf16(c, self.cond[0].weight, self.cond[0].bias, normalize=True, silu=True)
        cond = F.linear_bf16(cn, w_cond, b_cond, out_dtype=torch.float32)  # [rows, 6*dim] fp32
        x = x.contiguous().clone()
        h = attention(F.adaln(x, cond, 0, D, self.lns_scale), pairs, mask, multiplicity)
        F.gated_residual_(x, h, cond, 2 * D)
        h = self.transition(F.adaln(x, cond, 3 * D, 4 * D, self.lns_scale))
        F.gated_residual_(x, h, cond, 5 * D)
        return x
