"""Triangle multiplication modules with the reference's constructor / forward / state_dict contract.

Reference: ``_TriMulBase`` and ``TriangleMultiplicationFull`` in
src/bioemu2/biomoa/ops/triangle_multiplication.py:62-99, wrappers :370-395.  The parameters are the
same ``nn.LayerNorm`` / ``nn.Linear`` submodules under the same names, so checkpoints load unchanged;
the forward runs the sm_100a kernels (LayerNorm + gated projection, per-channel tcgen05 contraction,
LayerNorm + gated output projection).
"""
from __future__ import annotations

import torch
import torch.nn as nn
from torch import Tensor

from . import functional as F
from . import ieee, precision


def plain(module, cls) -> bool:
    """Whether calling ``module`` does what ``cls`` does and nothing besides (no subclass, no hook, no forward of its own), so
    that a call which covers several modules may stand for it."""
    if type(module) is not cls:
        return False
    own = module.__dict__
    return not own["_forward_hooks"] and not own["_forward_pre_hooks"] and "forward" not in own


def _watch_list(module: nn.Module):
    """Where a module tree keeps its parameters: (child dict, name, child) links and (parameter dict, name) slots."""
    links, slots, todo = [], [], [module]
    for m in todo:  # grows under way
        d = m._parameters
        slots += [(d, n) for n in d]
        d = m._modules
        if d:
            links += [(d, n, c) for n, c in d.items()]
            todo += [c for c in d.values() if c is not None]
    return links, slots


class PackedWeightsMixin:
    """Caches the bf16 kernel-layout copy of a module's parameters until one of them changes.

    The check runs on every forward, so it does not walk the module tree: it looks the parameters up through the
    dictionaries that hold them (a replaced submodule or parameter is seen there) and compares storage address and
    version counter -- addresses are unique over all devices."""

    _packed = None
    _packed_key = None
    _watch = None

    def __getstate__(self):
        """Copies and pickles of a module go without what is derived from its parameters (device addresses among it)."""
        kept = dict(self.__dict__)
        for name in ("_packed", "_packed_key", "_watch", "_split", "_split_key", "_side"):
            kept.pop(name, None)
        return kept

    def _pack_key(self):
        watch = self._watch
        if watch is not None:
            for d, n, c in watch[0]:
                if d.get(n) is not c:
                    watch = None
                    break
        if watch is None:
            watch = self.__dict__["_watch"] = _watch_list(self)  # (a module's own setattr looks for parameters first)
        key = []
        for d, n in watch[1]:
            p = d.get(n)
            if p is not None:
                key.append(p.data_ptr())
                key.append(p._version)
        return key

    def packed(self, build=None):
        """The packed copy; ``build`` replaces ``_build_packed`` when it has to be made anew."""
        key = self._pack_key()
        if self._packed is None or key != self._packed_key:
            with torch.no_grad():
                self.__dict__["_packed"] = self._build_packed() if build is None else build()
            self.__dict__["_packed_key"] = key
        return self._packed

    _split = None
    _split_key = None

    def split_weights(self):
        """The (hi | lo | hi) split copies of the projection weights used by the fp32-accurate forms."""
        key = self._pack_key()
        if self._split is None or key != self._split_key:
            with torch.no_grad():
                self._split = self._build_split()
            self._split_key = key
        return self._split


class TriangleMultiplication(PackedWeightsMixin, nn.Module):
    """``TriangleMultiplication(dim, mode)``; registry kwargs of the reference's variants are accepted.

    ``tile_size`` selects among the reference's backends (triangle_multiplication.py:170-198) and is ignored.
    ``matmul_precision="ieee"`` (triangle_multiplication.py:119-136) selects the fp32-accurate form for fp32 inputs,
    as does ``bioemu2_b200.precision.set_matmul_precision("ieee")``; the default is the bf16 tensor-core path.
    """

    def __init__(self, dim: int = 128, mode: str = "outgoing", tile_size: int | None = None,
                 matmul_precision: str | None = None, **kwargs) -> None:
        super().__init__()
        assert mode in ("outgoing", "incoming")
        if dim != 128:
            raise ValueError("bioemu2_b200 triangle multiplication is built for dim=128")
        self.mode = mode
        self.dim = dim
        self.matmul_precision = matmul_precision
        self.norm_in = nn.LayerNorm(dim, eps=1e-5)
        self.p_in = nn.Linear(dim, 2 * dim, bias=False)
        self.g_in = nn.Linear(dim, 2 * dim, bias=False)
        self.norm_out = nn.LayerNorm(dim)
        self.p_out = nn.Linear(dim, dim, bias=False)
        self.g_out = nn.Linear(dim, dim, bias=False)

    def _build_packed(self):
        return F.TriMulPacked(self.norm_in.weight, self.norm_in.bias, self.p_in.weight, self.g_in.weight,
                              self.norm_out.weight, self.norm_out.bias, self.p_out.weight, self.g_out.weight)

    def _build_split(self):
        p, g = self.p_in.weight, self.g_in.weight
        return ieee.SplitWeights(w_in=torch.cat([p[:128], g[:128], p[128:], g[128:]], dim=0),  # p and g of a, then of b
                                 w_p_out=self.p_out.weight, w_g_out=self.g_out.weight
                                 ).norms(norm_in=self.norm_in, norm_out=self.norm_out)

    def forward(self, x: Tensor, mask: Tensor) -> Tensor:
        """``x[B,N,N,dim]``, ``mask[B,N,N]`` -> update ``[B,N,N,dim]`` (no residual, like the reference)."""
        if precision.use_ieee(self.matmul_precision, x):
            return ieee.triangle_multiplication(x, mask, self, self.split_weights())
        return F.trimul(x, mask, self.packed(), incoming=self.mode == "incoming")

    def forward_residual(self, x: Tensor, mask: Tensor) -> Tensor:
        """``x + forward(x, mask)`` as a new tensor."""
        if precision.use_ieee(self.matmul_precision, x):
            return ieee.triangle_multiplication(x, mask, self, self.split_weights(), add_residual=True)
        return self.forward_residual_(x.clone(), mask)

    def forward_residual_(self, x: Tensor, mask: Tensor) -> Tensor:
        """``x += forward(x, mask)`` in place with the add fused into the output kernel; returns ``x``."""
        if precision.use_ieee(self.matmul_precision, x):
            return ieee.triangle_multiplication(x, mask, self, self.split_weights(), add_residual=True, out=x)
        return F.trimul(x, mask, self.packed(), incoming=self.mode == "incoming", add_residual=True, out=x)


class TriangleMultiplicationOutgoing(TriangleMultiplication):
    def __init__(self, dim: int = 128) -> None:
        super().__init__(dim=dim, mode="outgoing")


class TriangleMultiplicationIncoming(TriangleMultiplication):
    def __init__(self, dim: int = 128) -> None:
        super().__init__(dim=dim, mode="incoming")


_OWN_TRIMUL = (TriangleMultiplication, TriangleMultiplicationOutgoing, TriangleMultiplicationIncoming)


def native_trimul(module, mode: str) -> bool:
    """A triangle multiplication of that direction that a trunk's native call may stand for."""
    return type(module) in _OWN_TRIMUL and module.mode == mode and module.matmul_precision != "ieee"
