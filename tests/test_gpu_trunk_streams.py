"""The trunk's two streams, and threads that share a stream."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _trunk(blocks, seed):
    import bioemu2_b200 as b

    torch.manual_seed(seed)
    with torch.device("cuda"):
        return b.PairformerModule(384, 128, blocks).eval()


def _inputs(n, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    return (torch.randn(1, n, 384, device="cuda", generator=g), torch.randn(1, n, n, 128, device="cuda", generator=g),
            torch.rand(1, n, device="cuda", generator=g) > 0.1)


def test_a_call_that_fails_under_way_joins_its_side_stream():
    """A width that only the second block's transition kernel looks at: the first block's single track is on the side stream by
    then.  Without the join a capture could not end."""
    trunk, (s, z, mask) = _trunk(2, 1), _inputs(40, 1)
    with torch.no_grad():
        want = trunk(s, z, mask)  # packs the weights
    w, good = trunk.packed(), trunk.packed().array[1].transition_z.hidden
    graph = torch.cuda.CUDAGraph()
    w.array[1].transition_z.hidden = 300
    try:
        with torch.no_grad(), torch.cuda.graph(graph):
            s1 = s.clone()
            with pytest.raises(ValueError, match="hidden=300"):
                trunk.forward_into(s1, z, torch.empty_like(z), mask)
    finally:
        w.array[1].transition_z.hidden = good
    with torch.no_grad():
        again = trunk(s, z, mask)
    assert all(torch.equal(x, y) for x, y in zip(want, again))
