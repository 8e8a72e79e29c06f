"""The trunk's two streams, and threads that share a stream."""
import threading

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


@pytest.mark.parametrize("shared", [False, True])
def test_threads_on_one_stream(shared):
    """Two threads enqueue on the same stream at the same time, with a trunk each or with one between them: the results are those
    of calls one after the other."""
    trunks = [_trunk(2, 3)] * 2 if shared else [_trunk(2, 3), _trunk(2, 4)]
    inputs = [_inputs(72, 5), _inputs(40, 6)]
    with torch.no_grad():
        want = [t(*x) for t, x in zip(trunks, inputs)]
    torch.cuda.synchronize()
    start, got, errors = threading.Barrier(2), [[], []], []

    def work(i):
        try:
            with torch.no_grad():
                start.wait(30)
                for _ in range(20):
                    got[i].append(trunks[i](*inputs[i]))
        except Exception as exc:  # noqa: BLE001 - reported by the main thread
            errors.append(exc)

    threads = [threading.Thread(target=work, args=(i,)) for i in range(2)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    torch.cuda.synchronize()
    assert not errors, errors
    for w, runs in zip(want, got):
        assert len(runs) == 20
        for r in runs:
            assert torch.equal(r[0], w[0]) and torch.equal(r[1], w[1])
