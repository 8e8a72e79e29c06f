"""The sequence-trunk glue (pair initialisation, recycling, MSA module) and PairwiseConditioning on the GPU against the
golden vectors the reference's modules produced and against the CPU oracle."""
import os
import sys

import pytest
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.abspath(__file__)), "golden"))
import cases as C  # noqa: E402
import helpers as H  # noqa: E402
from gpu_util import assert_close  # noqa: E402
from oracle import pair_ops as O  # noqa: E402

pytestmark = pytest.mark.gpu


def _cuda(feats: dict) -> dict:
    return {k: v.cuda() for k, v in feats.items()}


# ------------------------------------------------------------------------------------------ kernels
def test_pair_outer_sum_is_exact():
    from bioemu2_b200 import functional as F

    g = torch.Generator().manual_seed(900)
    a, c = torch.randn(2, 37, 128, generator=g).cuda(), torch.randn(2, 53, 128, generator=g).cuda()
    extra = torch.randn(2, 37, 53, 128, generator=g).cuda()
    assert torch.equal(F.pair_outer_sum(a, c), a[:, :, None] + c[:, None])
    assert torch.equal(F.pair_outer_sum(a, c, extra), (a[:, :, None] + c[:, None]) + extra)


def test_add_rows_plain_and_broadcast():
    from bioemu2_b200 import functional as F

    g = torch.Generator().manual_seed(901)
    x = torch.randn(5, 33, 64, generator=g).cuda()
    y = torch.randn(5, 33, 64, generator=g).cuda()
    yb = torch.randn(33, 64, generator=g).cuda()
    assert torch.equal(F.add_rows(x, y), x + y)
    assert torch.equal(F.add_rows(x, yb), x + yb)
    assert torch.equal(F.add_rows(x, y.bfloat16()), x + y.bfloat16().float())
    x0 = x.clone()
    assert F.add_rows(x, yb, out=x) is x and torch.equal(x, x0 + yb)


@pytest.mark.parametrize("shape,nt", [((1, 1, 1), 33), ((2, 3, 37), 33), ((1, 5, 64), 5), ((1, 7, 11), 6), ((1, 0, 4), 33)])
@pytest.mark.parametrize("paired", [False, True])
def test_msa_features_are_the_rounded_concatenation(shape, nt, paired):
    """Whole columns (5 + 3, 6 + 2) and padded ones; fp32 features, and forms that go by copies, give the same bits."""
    from bioemu2_b200 import functional as F

    g = torch.Generator().manual_seed(910)
    msa = torch.randn(*shape, nt, generator=g).cuda()
    cols = [torch.randn(*shape, generator=g).cuda() for _ in range(2 + paired)]
    want = torch.cat([msa] + [c[..., None] for c in cols], -1).bfloat16()
    got = F.msa_features(msa, *cols)
    width = nt + len(cols)
    assert got.shape == (*shape, (width + 7) // 8 * 8) and got.dtype == torch.bfloat16
    assert torch.equal(got[..., :width], want) and not got[..., width:].any()
    for other in (F.msa_features(msa.transpose(0, 2).contiguous().transpose(0, 2), *cols),
                  F.msa_features(msa, cols[0].bfloat16().double(), *cols[1:])):
        assert torch.equal(other, got)


def test_two_source_layernorm_matches_the_concatenation():
    from bioemu2_b200 import functional as F

    g = torch.Generator().manual_seed(902)
    x1, x2 = torch.randn(301, 128, generator=g) * 2 + 0.5, torch.randn(301, 136, generator=g)
    w, b = torch.randn(264, generator=g), torch.randn(264, generator=g)
    want = torch.nn.functional.layer_norm(torch.cat([x1, x2], -1).double(), (264,), w.double(), b.double())
    got = F.rows2_to_bf16(x1.cuda(), x2.cuda(), w.cuda(), b.cuda())
    assert got.dtype == torch.bfloat16 and tuple(got.shape) == (301, 264)
    assert_close("rows2_to_bf16", got, want)
    one = F.rows_to_bf16(torch.cat([x1, x2], -1).cuda(), w.cuda(), b.cuda())
    assert torch.equal(got, one)  # same arithmetic as the one-source kernel on the materialised concatenation


# ------------------------------------------------------------------------------------------ PairwiseConditioning
def _cond(w):
    import bioemu2_b200 as b

    m = b.PairwiseConditioning(token_z=128, dim_token_rel_pos_feats=128).eval()
    m.load_state_dict(w, strict=True)
    return m.cuda()


def test_pairwise_conditioning_golden():
    golden = torch.load(C.GOLDEN_PATH)
    case = C.CASES["pairwise_conditioning"]()
    mod = _cond(case["w"])
    z, rel = case["z"].cuda(), case["rel"].cuda()
    z0 = z.clone()
    with torch.no_grad():
        out = mod(z, rel)
    assert out.dtype == torch.float32 and torch.equal(z, z0)
    assert_close("pairwise_conditioning_golden", out, golden["pairwise_conditioning"]["output"], atol=4e-2)


@pytest.mark.parametrize("N", [72, 200])
def test_pairwise_conditioning_vs_oracle(N):
    g = torch.Generator().manual_seed(910 + N)
    w = H.pairwise_conditioning_weights(g)
    z = torch.randn(1, N, N, 128, generator=g)
    rel = torch.randn(1, N, N, 128, generator=g)
    ref = O.pairwise_conditioning(z.double(), rel.double(), {k: v.double() for k, v in w.items()})
    with torch.no_grad():
        out = _cond(w)(z.cuda(), rel.cuda())
    assert_close(f"pairwise_conditioning_N{N}", out, ref, atol=4e-2)


@pytest.mark.parametrize("B,n_i,n_j,transitions,factor,dtype", [
    (1, 1, 1, 2, 2, torch.float32),       # a single row
    (1, 8, 16, 1, 2, torch.float32),      # one whole tile, one transition
    (2, 9, 15, 2, 2, torch.bfloat16),     # a tile and a part of one
    (1, 160, 148, 2, 2, torch.bfloat16),  # a second tile for some CTAs
    (1, 290, 131, 2, 1, torch.float32),   # three tiles a CTA, hidden padded to 256
    (1, 12, 12, 2, 4, torch.float32),     # hidden 512 and three transitions: the passes one by one
    (1, 12, 12, 3, 2, torch.float32),
])
def test_pairwise_conditioning_shapes(B, n_i, n_j, transitions, factor, dtype):
    import bioemu2_b200 as b
    from bioemu2_b200 import _lib

    g = torch.Generator().manual_seed(915 + n_i)
    w = H.pairwise_conditioning_weights(g, num_transitions=transitions, factor=factor)
    z, rel = (torch.randn(B, n_i, n_j, 128, generator=g).to(dtype) for _ in range(2))
    ref = O.pairwise_conditioning(z.double(), rel.double(), {k: v.double() for k, v in w.items()}, transitions)
    m = b.PairwiseConditioning(128, 128, num_transitions=transitions, transition_expansion_factor=factor).eval()
    m.load_state_dict(w, strict=True)
    with torch.no_grad():
        out = m.cuda()(z.cuda(), rel.cuda())
    assert _lib.device_status() == 0 and out.dtype == torch.float32
    assert_close(f"pairwise_conditioning_{B}x{n_i}x{n_j}_{transitions}_{factor}_{dtype}", out, ref, atol=4e-2)


@pytest.mark.parametrize("transitions", [1, 2, 3])
def test_pairwise_conditioning_of_rows_far_from_zero(transitions):
    """Rows of z whose mean is two thousand times their deviation: the LayerNorms in between have to find the deviation (three
    transitions go pass by pass).  Channel 0 of the input's LayerNorm is constant and adds 1024 to all of z, exactly; z itself then
    has 2^-13 of a unit, the operands bf16's 2^-9 as ever."""
    import bioemu2_b200 as b

    g = torch.Generator().manual_seed(917)
    w = H.pairwise_conditioning_weights(g, num_transitions=transitions)
    w["dim_pairwise_init_proj.0.weight"][0], w["dim_pairwise_init_proj.0.bias"][0] = 0.0, 2.0
    w["dim_pairwise_init_proj.1.weight"][:, 0] = 512.0
    z, rel = (torch.randn(1, 20, 13, 128, generator=g) for _ in range(2))
    ref = O.pairwise_conditioning(z.double(), rel.double(), {k: v.double() for k, v in w.items()}, transitions)
    m = b.PairwiseConditioning(128, 128, num_transitions=transitions).eval()
    m.load_state_dict(w, strict=True)
    with torch.no_grad():
        out = m.cuda()(z.cuda(), rel.cuda())
    assert_close(f"pairwise_conditioning_far_{transitions}", out.double() - 1024, ref - 1024, atol=4e-2)


# ------------------------------------------------------------------------------------------ MSA module, trunk
def test_msa_module_golden():
    import bioemu2_b200 as b

    golden = torch.load(C.GOLDEN_PATH)
    case = C.CASES["msa_module"]()
    mod = b.PairMixerMSAModule(token_s=384, msa_s=64, token_z=128, s_input_dim=case["emb"].shape[-1],
                               msa_blocks=case["blocks"], use_paired_feature=True).eval()
    mod.load_state_dict(case["w"], strict=True)
    mod.cuda()
    f = _cuda(case["feats"])
    with torch.no_grad():
        s, z = mod(None, case["z"].cuda(), case["emb"].cuda(), f["msa"], f["msa_mask"], f["has_deletion"],
                   f["deletion_value"], f["msa_paired"], f["token_pad_mask"])
    assert s is None
    # two MSA blocks = eight residual updates of the pair tensor
    assert_close("msa_module_golden", z, golden["msa_module"]["output"], atol=4e-2)


def _embedder(case):
    import bioemu2_b200 as b

    mod = b.PairMixerSequenceEmbedder(token_s=384, token_z=128, s_input_dim=case["s_inputs"].shape[-1], msa_s=64,
                                      msa_blocks=case["msa_blocks"], num_blocks=case["num_blocks"],
                                      use_paired_feature=True, use_unconditional_branch=True).eval()
    mod.load_state_dict(case["w"], strict=True)
    return mod.cuda()


@pytest.mark.parametrize("name", ["sequence_trunk", "sequence_trunk_unconditional"])
def test_sequence_trunk_golden(name):
    """One recycle (two passes through the MSA block and the PairMixer block) and the unconditional branch; the
    encoders' pair terms enter through ``feats["pair_init_terms"]``."""
    golden = torch.load(C.GOLDEN_PATH)
    case = C.CASES[name]()
    mod = _embedder(case)
    feats = dict(_cuda(case["feats"]), pair_init_terms=case["pair_terms"].cuda())
    with torch.no_grad():
        s, z = mod(case["s_inputs"].cuda(), feats, num_steps_recycle=case["recycles"], unconditional=case["unconditional"])
    want = golden[name]["output"]
    nz = z.numel()
    assert s.dtype == torch.float32 and z.dtype == torch.float32
    assert_close(f"{name}_z", z.flatten(), want[:nz], atol=4e-2)
    assert_close(f"{name}_s", s.flatten(), want[nz:], atol=4e-2)


def test_sequence_trunk_encoders_are_called_like_the_reference():
    """Feature encoders assigned to the module are called with the reference's keyword arguments and summed."""
    import bioemu2_b200 as b

    case = C.CASES["sequence_trunk_unconditional"]()
    mod = _embedder(case)
    seen = {}

    class RelPos(torch.nn.Module):
        def forward(self, asym_id, entity_id, residue_index, sym_id):
            seen["rel_pos"] = (asym_id, entity_id, residue_index, sym_id)
            return case["pair_terms"].cuda() * 0.25

    class Bonds(torch.nn.Module):
        def forward(self, token_bonds):
            seen["token_bonds"] = token_bonds
            return case["pair_terms"].cuda() * 0.75

    feats = dict(_cuda(case["feats"]), asym_id=1, entity_id=2, residue_index=3, sym_id=4, token_bonds=5)
    with torch.no_grad():
        want = mod(case["s_inputs"].cuda(), dict(feats, pair_init_terms=case["pair_terms"].cuda()), unconditional=True)
        mod.rel_pos, mod.token_bonds = RelPos(), Bonds()
        got = mod(case["s_inputs"].cuda(), feats, unconditional=True)
    assert seen == {"rel_pos": (1, 2, 3, 4), "token_bonds": 5}
    assert "rel_pos" in dict(mod.named_children())
    torch.testing.assert_close(got[1], want[1], atol=1e-5, rtol=1e-5)
    assert isinstance(mod, b.PairMixerSequenceEmbedder)


@pytest.mark.parametrize("n,rows", [(256, 128), (100, 37)])
def test_two_passes_are_equal(n, rows):
    """Enough tiles that every CTA of a product reuses its staging tiles, whose stores have to be read out first."""
    import bioemu2_b200 as b

    g = torch.Generator(device="cuda").manual_seed(n)
    rand = lambda *s: torch.rand(*s, device="cuda", generator=g)  # noqa: E731
    with torch.device("cuda"):
        mod = b.PairMixerSequenceEmbedder(384, 128, 456, msa_s=64, msa_blocks=1, num_blocks=1).eval()
    tok = torch.ones(1, n, dtype=torch.bool, device="cuda")
    tok[:, n - 7:] = False
    feats = {"msa": torch.nn.functional.one_hot((rand(1, rows, n) * 33).long(), 33).float(), "token_pad_mask": tok,
             "msa_mask": tok[:, None] & (rand(1, rows, n) > 0.1), "has_deletion": (rand(1, rows, n) < 0.2).float(),
             "deletion_value": rand(1, rows, n), "msa_paired": (rand(1, rows, n) < 0.5).float()}
    x = rand(1, n, 456) - 0.5
    with torch.no_grad():
        first = mod(x, feats, num_steps_recycle=1)
        for _ in range(8):
            again = mod(x, feats, num_steps_recycle=1)
            assert all(torch.equal(p, q) for p, q in zip(first, again))


def test_sequence_trunk_argument_errors():
    case = C.CASES["sequence_trunk"]()
    mod = _embedder(case)
    feats = _cuda(case["feats"])
    with pytest.raises(ValueError, match="non-negative"):
        mod(case["s_inputs"].cuda(), feats, num_steps_recycle=-1)
    mod.use_unconditional_branch = False
    with pytest.raises(ValueError, match="use_unconditional_branch"):
        mod(case["s_inputs"].cuda(), feats, unconditional=True)


def test_context_parallel_wrappers_of_the_per_pair_glue():
    """The per-pair ops need no exchange: the wrappers run the serial kernels on a rank's block, so a block of the
    full result equals the result on the block."""
    import bioemu2_b200 as b
    from bioemu2_b200.context_parallel import ops

    g = torch.Generator().manual_seed(920)
    w = H.pairwise_conditioning_weights(g)
    serial = _cond(w)
    z = torch.randn(1, 96, 96, 128, generator=g).cuda()
    rel = torch.randn(1, 96, 96, 128, generator=g).cuda()
    with torch.no_grad():
        full = serial(z, rel)
        blk = ops.DistributedPairwiseConditioning(serial)(z[:, 48:, :40].contiguous(), rel[:, 48:, :40].contiguous())
        assert torch.equal(blk, full[:, 48:, :40])
        tiled = ops.LayerNormLinearParamsReplicatedTiled(serial.dim_pairwise_init_proj)
        assert sorted(tiled.state_dict()) == ["0.bias", "0.weight", "1.weight"]
        proj = tiled(z, rel)
        ln = serial.dim_pairwise_init_proj[0]
        want = torch.nn.functional.linear(
            torch.nn.functional.layer_norm(torch.cat([z, rel], -1).double(), (256,), ln.weight.double(), ln.bias.double()),
            serial.dim_pairwise_init_proj[1].weight.double())
        assert_close("ln_linear_tiled", proj, want)
    with pytest.raises(RuntimeError, match="forward-only"):
        tiled(z, rel)
    assert isinstance(serial, b.PairwiseConditioning)
