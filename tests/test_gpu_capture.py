"""The flop-EV chain and the flop matrices in a captured graph: a replay works
from what the graph and its caller keep."""
import ctypes
import importlib

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


@pytest.mark.parametrize("mode", [0, 1])
def test_flop_matrices_replay(mtt, cuda, mode):
    import torch
    pf = importlib.import_module("mtt-gpu-solver_b200.preflop")
    lib = importlib.import_module("mtt-gpu-solver_b200._lib").lib()
    host = np.ascontiguousarray(mtt.canonical_flops()[::60, :3])
    flops = torch.from_numpy(host).to(cuda)
    out = torch.zeros(len(host), 169, 169, device=cuda)
    ptr = lambda x: ctypes.c_void_p(x)

    def call():
        st = lib.mtt_pf_flop_class_matrices(mode, ptr(flops.data_ptr()), len(host), ptr(out.data_ptr()),
                                            ptr(torch.cuda.current_stream().cuda_stream))
        assert st == 0
        return [out]

    _replayed(call)
    assert torch.equal(out, pf.flop_class_matrices(host, mode))
