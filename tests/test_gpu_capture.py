"""The flop-EV chain in a captured graph: a replay works from what the graph and
its caller keep."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _replayed(call):
    """Results of a call and of two replays of it, other calls of other host data between."""
    import torch
    want = [t.clone() for t in call()]
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        got = call()
    for _ in range(2):
        for t in got:
            t.fill_(7)
        churn = [np.full(4096, 255, np.uint8) for _ in range(64)]
        graph.replay()
        torch.cuda.synchronize()
        assert all(torch.equal(a, b) for a, b in zip(want, got))
        del churn


@pytest.mark.parametrize("n", [1, 70])
def test_flop_ev_replays(mtt, cuda, n):
    import torch
    flops = torch.from_numpy(np.ascontiguousarray(mtt.canonical_flops()[::25][:n, :3])).to(cuda)
    _replayed(lambda: mtt.flop_ev(flops))
    _replayed(lambda: [mtt.ev_dump(flops)])
