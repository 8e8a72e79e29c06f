"""Arguments that a call cannot serve are refused on the host, before a kernel is given their addresses (no GPU needed)."""
from types import SimpleNamespace

import pytest
import torch

from bioemu2_b200 import _lib
from bioemu2_b200 import functional as F
from bioemu2_b200 import ieee
from bioemu2_b200.sequence_trunk import PairMixerMSAModule


@pytest.mark.parametrize("shape,mask,exc", [
    ((1, 20, 12, 128), (1, 20, 12), ValueError),      # not square
    ((1, 12, 12, 64), (1, 12, 12), ValueError),       # another width
    ((12, 12, 128), (12, 12), ValueError),
    ((2, 12, 12, 128), (1, 12, 12), ValueError),
    ((1, 12, 12, 128), (1, 12, 11), ValueError),
    ((1, 12, 12, 128), (1, 12, 12), RuntimeError),    # on the host
])
@pytest.mark.parametrize("add_residual", [False, True])
def test_accurate_triangle_multiplication(shape, mask, exc, add_residual):
    x = torch.zeros(shape)
    with pytest.raises(exc, match="CUDA tensors" if exc is RuntimeError else "expected x|mask shape"):
        ieee.triangle_multiplication(x, torch.ones(mask, dtype=torch.bool), SimpleNamespace(mode="outgoing"), SimpleNamespace(),
                                     add_residual, out=x if add_residual else None)


@pytest.mark.parametrize("native", [False, True])
@pytest.mark.parametrize("width,exc", [(192, ValueError), (64, ValueError), (128, RuntimeError)])
def test_accurate_transition(width, exc, native):
    ws = SimpleNamespace(w12=torch.empty(512, 3 * 128), w3=torch.empty(128, 3 * 256), norm_w=None, norm_b=None, native=native)
    with pytest.raises(exc, match="CUDA tensors" if exc is RuntimeError else "expected x"):
        ieee.transition(torch.zeros(5, width), None, None, None, None, ws)


class _OnDevice(torch.Tensor):
    """A tensor that says it is on the GPU."""

    is_cuda = property(lambda self: True)


@pytest.mark.parametrize("call", [
    lambda d, h: F.ln_linear(d(4, 128), h(4, 128), None, None, d(128, 256).bfloat16()),
    lambda d, h: F.ln_linear(d(4, 128), None, None, None, d(128, 128).bfloat16(), residual=h(4, 128)),
    lambda d, h: F.outer_product_mean(d(1, 3, 4, 64), d(1, 3, 4), None, residual=h(1, 4, 4, 128)),
    lambda d, h: F.trunk_(d(1, 4, 4, 128), d(1, 4, 4, 128), None, None, h(1, 4, 4), None),
    lambda d, h: F.trunk_(d(1, 4, 4, 128), d(1, 4, 4, 128), d(1, 4, 64), h(1, 4), None, None),
    lambda d, h: F.trunk_(d(1, 4, 4, 128), d(1, 4, 4, 128), h(1, 4, 64), d(1, 4), None, None),
    lambda d, h: F.cond_layer(None, d(1, 4, 64), h(1, 4, 4, 128), None, d(1, 4, 64), d(1, 4)),
    lambda d, h: F.TransitionGenericPacked(None, None, d(64, 64), d(64, 64), h(64, 64)),
    lambda d, h: ieee.split(h(4, 64), 0),
], ids=["second_source", "residual", "opm_residual", "pair_mask", "token_mask", "single", "pairs", "weights", "split"])
def test_one_tensor_on_the_host(call):
    with pytest.raises(RuntimeError, match="CUDA tensors"):
        call(lambda *s: torch.zeros(s).as_subclass(_OnDevice), lambda *s: torch.zeros(s))


def _msa(paired: bool, **kw):
    m = PairMixerMSAModule(64, 64, 128, 16, 1, use_paired_feature=paired)
    feats = dict(emb=torch.zeros(1, 5, 16), msa=torch.zeros(1, 3, 5, 33), has_deletion=torch.zeros(1, 3, 5),
                 deletion_value=torch.zeros(1, 3, 5), msa_paired=torch.zeros(1, 3, 5) if paired else None)
    return m.embed_msa(**{**feats, **kw})


@pytest.mark.parametrize("tokens", [None, slice(0, 5)])
def test_msa_embedding_without_its_paired_feature(tokens):
    """With 33 token columns both widths are padded to 40, so the product alone would not notice."""
    with pytest.raises(TypeError, match="msa_paired"):
        _msa(True, msa_paired=None, tokens=tokens)
    for paired in (True, False):
        with pytest.raises(RuntimeError, match="CUDA tensors"):
            _msa(paired, tokens=tokens)


@pytest.mark.parametrize("shape", [(3, 5, 33), (1, 1, 3, 5, 33)])
def test_msa_embedding_of_another_rank(shape):
    with pytest.raises(ValueError, match="msa must be"):
        _msa(False, msa=torch.zeros(shape), has_deletion=torch.zeros(shape[:-1]), deletion_value=torch.zeros(shape[:-1]))


def test_msa_feature_columns_given_as_numbers_or_rows():
    msa = torch.randn(2, 3, 5, 6)
    got = F.msa_features(msa, True, torch.full((5,), 0.5), 0.25)
    want = torch.cat([msa, torch.tensor([1.0, 0.5, 0.25]).expand(2, 3, 5, 3), torch.zeros(2, 3, 5, 7)], -1)
    assert torch.equal(got, want.bfloat16())


@pytest.mark.parametrize("width,heads", [(768, 16), (192, 16), (384, 8)])
def test_trunk_single_track_of_another_width(width, heads):
    w = F.TrunkPacked([])
    w.single = {(384, 16)}
    z = torch.zeros(1, 4, 4, 128).as_subclass(_OnDevice)
    s, mask = torch.zeros(1, 4, width).as_subclass(_OnDevice), torch.ones(1, 4).as_subclass(_OnDevice)
    with pytest.raises(ValueError, match="do not match the blocks"):
        F.trunk_(z, z, s, mask, None, w, heads)


def test_trunk_single_track_widths_come_from_every_block():
    def block(c_s, cols, heads):
        return {"attention": SimpleNamespace(c_s=c_s, H=heads, struct=_lib.ApbWeights()),
                "transition_s": SimpleNamespace(cols=cols, struct=_lib.SwigluWeights())}

    assert F.TrunkPacked([block(384, 384, 16)] * 2).single == {(384, 16)}
    assert F.TrunkPacked([{}]).single == set()
    assert len(F.TrunkPacked([block(384, 384, 16), block(384, 384, 8)]).single) == 2
    assert len(F.TrunkPacked([block(384, 768, 16)]).single) == 2
