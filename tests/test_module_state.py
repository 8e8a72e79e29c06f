"""What a module keeps between calls, and what it does not (no GPU needed)."""
import torch

from bioemu2_b200 import _lib
from bioemu2_b200 import functional as F


def test_conditioned_layer_reads_its_scale_on_every_call(monkeypatch):
    import bioemu2_b200 as b

    m = b.ConditionedTransformerLayer(dim=64, dim_pairwise=128, dim_cond=64, heads=4, transition_hidden=128, lns_scale=0.5)
    kept = _lib.CondLayer()
    kept.dim_cond = 64
    monkeypatch.setattr(m, "packed", lambda: (None, None, (kept, ())))
    monkeypatch.setattr(F, "cond_layer", lambda layer, *args: layer.lns_scale)
    args = torch.zeros(1, 8, 64), torch.zeros(1, 8, 8, 128), torch.zeros(1, 8, 64)
    assert m(*args) == 0.5
    m.lns_scale = 0.25
    assert m(*args) == 0.25
