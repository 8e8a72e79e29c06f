"""Contiguous views that start 16 bytes into a larger buffer give what an aligned tensor gives."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _view(t):
    lead = 16 // t.element_size()
    v = torch.empty(lead + t.numel(), dtype=t.dtype, device=t.device)[lead:].view(t.shape).copy_(t)
    assert v.is_contiguous() and v.data_ptr() % 32 == 16
    return v


@pytest.mark.parametrize("kind", ["pairformer", "pairmixer", "pairmixer_accurate", "conditioned", "transition"])
def test_offset_views(kind):
    import bioemu2_b200 as b

    g = torch.Generator(device="cuda").manual_seed(5)
    randn = lambda *s: torch.randn(*s, device="cuda", generator=g)  # noqa: E731
    tok = torch.ones(1, 24, dtype=torch.bool, device="cuda")
    pm = tok[:, :, None] & tok[:, None, :]
    with torch.device("cuda"):
        if kind == "pairformer":
            m, moved, rest = b.PairformerModule(384, 128, 2), [randn(1, 24, 384), randn(1, 24, 24, 128)], [tok]
        elif kind == "pairmixer":
            m, moved, rest = b.PairMixerModule(384, 128, 2), [None, randn(1, 24, 24, 128)], [pm]
        elif kind == "pairmixer_accurate":
            m, moved, rest = b.PairMixerLayer(384, 128), [None, randn(1, 24, 24, 128)], [pm]
        elif kind == "conditioned":
            m = b.ConditionedTransformerLayer(dim=384, dim_pairwise=128, dim_cond=384, heads=16, transition_hidden=768)
            moved, rest = [randn(1, 24, 384)], [randn(1, 24, 24, 128), randn(1, 24, 384), tok]
        else:  # bf16 rows that are a product's operand as they are
            m, moved, rest = b.Transition(384, 768, use_norm=False), [randn(24, 384).bfloat16()], []
    m.eval()
    kept = [None if t is None else t.clone() for t in moved]
    with torch.no_grad(), b.precision.matmul_precision("ieee" if kind.endswith("accurate") else "bf16"):
        want = m(*moved, *rest)
        views = [None if t is None else _view(t) for t in moved]
        got = m(*views, *rest)
    for w, v in zip(*((r,) if torch.is_tensor(r) else r for r in (want, got))):
        assert w is v is None or torch.equal(w, v)
    for k, v in zip(kept, views):
        assert k is v is None or torch.equal(k, v)  # the inputs stay as they were


@pytest.mark.parametrize("windowed", [False, True])
def test_conditioned_layer_takes_conditioning_by_rows_and_masks_by_windows(windowed):
    import bioemu2_b200 as b

    g = torch.Generator(device="cuda").manual_seed(6)
    randn = lambda *s: torch.randn(*s, device="cuda", generator=g)  # noqa: E731
    kw = dict(is_sliding_window=True, window_queries=32, window_keys=128) if windowed else {}
    with torch.device("cuda"):
        m = b.ConditionedTransformerLayer(128, 16 if windowed else 128, 128, 4, 256, **kw).eval()
    x, c = randn(2, 64, 128), randn(2, 64, 128)
    pairs = randn(1, 2, 32, 128, 16) if windowed else randn(1, 64, 64, 128)
    mask = torch.rand(1, 64, device="cuda", generator=g) > 0.1
    with torch.no_grad():
        want = m(x, pairs, c, mask, 2)
        assert torch.equal(m(x, pairs, c.view(128, 128), mask, 2), want)
        for shape in ((2, 32), (1, 2, 32)):
            if windowed:
                assert torch.equal(m(x, pairs, c, mask.view(shape), 2), want)
            else:
                with pytest.raises(ValueError):
                    m(x, pairs, c, mask.view(shape), 2)
        with pytest.raises(ValueError):
            m(x, pairs, c[:1], mask, 2)
