"""What a module keeps between calls, and what it does not (no GPU needed)."""
import copy
import gc
import pickle
import threading
from types import SimpleNamespace

import pytest
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


@pytest.mark.parametrize("make", [lambda b: b.Transition(128, 512), lambda b: b.PairwiseConditioning(128, 128),
                                  lambda b: b.PairMixerModule(384, 128, 1)])
def test_a_module_that_has_packed_its_weights_can_be_copied(make):
    import bioemu2_b200 as b

    m = make(b)
    for child in m.modules():
        if hasattr(child, "packed"):
            child._pack_key()
            child._packed, child._split = (SimpleNamespace(struct=_lib.TransitionWeights(1, 2, 3, 4, 512)) for _ in range(2))
    for other in (copy.deepcopy(m), pickle.loads(pickle.dumps(m))):
        assert [k for k, _ in other.named_parameters()] == [k for k, _ in m.named_parameters()]
        for child, kept in zip(other.modules(), m.modules()):
            if hasattr(child, "packed"):
                assert child._packed is None and child._split is None and kept._packed is not None
                assert child._pack_key() != kept._pack_key()


@pytest.mark.parametrize("hidden", [256, 512, 200, 64, 448])
def test_fused_transition_weights(monkeypatch, hidden):
    """Alternating blocks of 64 rows of fc1 and fc2, padded with zeros to the kernel's width; whole widths are few segments, for
    packing them is most of what a first pass on new weights costs the host."""
    parts = []

    def build(pk, device):
        out = torch.zeros(pk.size)
        for t, off, groups, group, pitch, stride, scale in pk.parts:
            parts.append(t)
            for k in range(groups if t is not None else 0):
                out[off + k * stride:off + k * stride + group] = scale * t.reshape(-1)[k * group:(k + 1) * group]
        return out

    monkeypatch.setattr(F._Pack, "build", build)
    fc1, fc2, fc3 = torch.randn(hidden, 128), torch.randn(hidden, 128), torch.randn(128, hidden)
    w = F.TransitionPacked(None, None, fc1, fc2, fc3)
    width = 256 if hidden <= 256 else 512
    wide = torch.zeros(2, width, 128)
    wide[0, :hidden], wide[1, :hidden] = fc1, fc2
    assert torch.equal(w.w13.view(width // 64, 2, 64, 128), wide.view(2, width // 64, 64, 128).transpose(0, 1))
    assert torch.equal(w.w3[:, :hidden], fc3) and not w.w3[:, hidden:].any()
    assert len(parts) == 3 or hidden != width


def test_workspaces_of_threads_are_apart_and_go_back_together(monkeypatch):
    monkeypatch.setattr(F, "_stream", lambda: 7)
    cpu, seen, go, done = torch.device("cpu", 0), {}, threading.Event(), threading.Event()

    def work():
        seen["first"] = F.workspace(4096, cpu)
        done.set()
        go.wait(30)
        seen["again"] = F.workspace(100, cpu)

    mine = F.workspace(4096, cpu)
    thread = threading.Thread(target=work)
    thread.start()
    assert done.wait(30)
    assert seen["first"].data_ptr() != mine.data_ptr() and seen["first"].data_ptr() % 1024 == 0
    assert F.workspace(100, cpu) is mine
    F.release_workspaces()
    go.set()
    thread.join()
    assert seen["again"] is not seen["first"] and F.workspace(100, cpu) is not mine
    del seen["again"]
    gc.collect()
    assert all(b is F._WORKSPACES.buffers for b in F._WORKSPACES.of_all_threads.values())  # the thread's went with it
    F.release_workspaces()


class _Adds(torch.nn.Module):
    """Stands where one of the package's modules stood."""

    matmul_precision = None

    def __init__(self, keeps=None):
        super().__init__()
        self.keeps, self._bias_cache, self._fused = keeps, None, False

    def forward(self, x, *args):
        return torch.ones_like(x)

    def forward_residual(self, x, *args):
        return x + 1

    def forward_residual_(self, x, *args):
        return x.add_(1)


def _refuse(*args, **kwargs):
    raise AssertionError("a native call")


@pytest.mark.parametrize("keep", [False, True])
def test_trunks_run_the_modules_that_were_put_into_them(monkeypatch, keep):
    """``keep``: the stand-in holds the old module, so the parameters are the ones the stack knows."""
    import bioemu2_b200 as b

    monkeypatch.setattr(_lib, "raise_if_device_wait", lambda: None)
    for name in ("trunk_", "trunk_blocks_"):
        monkeypatch.setattr(F, name, _refuse)
    s, z = torch.zeros(1, 4, 384), torch.zeros(1, 4, 4, 128)
    tok = torch.ones(1, 4, dtype=torch.bool)
    for trunk, mask in ((b.PairMixerModule(384, 128, 2), tok[:, :, None] & tok[:, None, :]), (b.PairformerModule(384, 128, 2), tok)):
        trunk.eval()
        trunk._pack_key()
        updates = 0
        for layer in trunk.layers:
            for name, child in list(layer.named_children()):
                updates += name not in ("attention", "transition_s")
                setattr(layer, name, _Adds(child if keep else None))
        with torch.no_grad():
            got = trunk(s, z, mask)
        assert torch.equal(got[1], torch.full_like(z, updates)) and not z.any()

    layer = b.PairMixerLayer(384, 128).eval()
    for name, child in list(layer.named_children()):
        setattr(layer, name, _Adds())
    assert torch.equal(layer(s, z, None)[1], z + 3)


@pytest.mark.parametrize("change", ["mode", "width", "subclass"])
def test_trunk_blocks_that_differ_run_by_themselves(monkeypatch, change):
    import bioemu2_b200 as b

    class Own(b.PairMixerLayer):
        pass

    trunk, ran = b.PairMixerModule(384, 128, 2).eval(), []
    assert all(trunk._native(m) for m in trunk.layers)
    if change == "mode":
        trunk.layers[1].tri_mul_in = b.TriangleMultiplicationOutgoing(128)
    elif change == "width":
        trunk.layers[1].transition_z = b.Transition(128, 1024)
    else:
        trunk.layers[1] = Own(384, 128)
    for name in ("trunk_", "trunk_blocks_"):
        monkeypatch.setattr(F, name, _refuse)
    monkeypatch.setattr(b.PairMixerLayer, "forward_", lambda self, z, mask: ran.append(self))
    monkeypatch.setattr(_lib, "raise_if_device_wait", lambda: None)
    trunk(None, torch.zeros(1, 4, 4, 128), torch.ones(1, 4, 4, dtype=torch.bool))
    assert ran == list(trunk.layers)


@pytest.mark.parametrize("windowed", [False, True])
def test_conditioned_layer_runs_the_modules_that_were_put_into_it(monkeypatch, windowed):
    import bioemu2_b200 as b

    def layer():
        kw = dict(is_sliding_window=True, window_queries=32, window_keys=128) if windowed else {}
        m = b.ConditionedTransformerLayer(128, 16 if windowed else 128, 128, 4, 512, **kw)
        kept = _lib.CondLayer()
        kept.dim_cond, kept.window_queries, kept.window_keys, kept.dim_pairwise = 128, 32, 128, 16
        monkeypatch.setattr(m, "packed", lambda: (None, None, (kept, ())))
        monkeypatch.setattr(m, "_forward", lambda *args: "by modules")
        return m

    monkeypatch.setattr(F, "cond_layer", lambda *args: "one call")
    pairs = torch.zeros(1, 1, 32, 128, 16) if windowed else torch.zeros(1, 32, 32, 128)
    args = torch.zeros(1, 32, 128), pairs, torch.zeros(1, 32, 128)
    assert layer()(*args) == "one call"
    for hooked in ("transition", "attention", "attention.pair_bias_attn" if not windowed else "attention.attention_layer"):
        m = layer()
        handle = m.get_submodule(hooked).register_forward_hook(lambda *a: None)
        assert m(*args) == "by modules"
        handle.remove()
        assert m(*args) == "one call"
    m = layer()
    with m.transition.register_forward_hook(lambda *a: None):  # what is packed meanwhile serves both ways
        monkeypatch.setattr(F, "_require_cuda", lambda *tensors: None)
        monkeypatch.setattr(F._Pack, "build", lambda pk, device: torch.zeros(pk.size))
        assert b.ConditionedTransformerLayer._build_packed(m)[2] is not None and m(*args) == "by modules"
    m = layer()
    m.transition = _Adds()
    assert m(*args) == "by modules"
    m = layer()
    m.attention = _Adds()
    assert m(*args) == "by modules"


def test_msa_layer_runs_the_outer_product_mean_that_was_put_into_it(monkeypatch):
    import bioemu2_b200 as b

    monkeypatch.setattr(F, "add_rows", lambda x, y: x + y)
    m = b.PairMixerMSALayer(384, 64, 128).eval()
    for name, child in list(m.named_children()):
        setattr(m, name, _Adds())
    m.outer_product_mean.forward = lambda msa, mask: torch.full((1, 4, 4, 128), 7.0)
    z = torch.zeros(1, 4, 4, 128)
    _, got, _ = m(None, z, torch.zeros(1, 3, 4, 64), torch.ones(1, 4, 4), torch.ones(1, 3, 4))
    assert torch.equal(got, z + 10)


@pytest.mark.parametrize("own", [False, True])
def test_embedder_runs_the_msa_module_that_was_put_into_it(monkeypatch, own):
    """The package's own module is handed the embedding of all recycling steps, another one the arguments it has always had."""
    import bioemu2_b200 as b

    calls, embedded = [], []

    class Msa(torch.nn.Module):
        def forward(self, s, z, emb, msa, msa_mask, has_deletion, deletion_value, msa_paired, token_pad_mask):
            calls.append((msa, token_pad_mask))
            return s, z

    class Mixer(torch.nn.Module):
        def forward(self, s, z, pair_mask):
            return s, z

    m = b.PairMixerSequenceEmbedder(64, 128, 16, msa_blocks=1, num_blocks=1).eval()
    m.pairmixer_module = Mixer()
    monkeypatch.setattr(m, "initial_embeddings", lambda s_inputs, feats: (torch.zeros(1, 4, 64), torch.zeros(1, 4, 4, 128)))
    monkeypatch.setattr(m, "_recycle", lambda x, x_init, norm, name: x_init)
    if own:
        monkeypatch.setattr(m.msa_module, "embed_msa", lambda *args: embedded.append(args) or "m")
        m.msa_module.layers = torch.nn.ModuleList([Msa()])
        m.msa_module.layers[0].forward = lambda s, z, m, *args: calls.append(m) or (s, z, m)
    else:
        m.msa_module = Msa()
    feats = {k: k for k in ("msa", "msa_mask", "has_deletion", "deletion_value", "msa_paired")}
    feats["token_pad_mask"] = torch.ones(1, 4)
    m(torch.zeros(1, 4, 16), feats, num_steps_recycle=2)
    assert len(calls) == 3 and len(embedded) == own
    assert calls == ["m"] * 3 if own else all(c[0] == "msa" and c[1] is feats["token_pad_mask"] for c in calls)
