"""The preflop solve, which runs on the legacy default stream unless told
otherwise, called from another current stream: its results and the copies of
its inputs need no wait of the caller's own."""
import importlib

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_preflop_solve_from_a_side_stream(mtt, cuda):
    import torch
    pf = importlib.import_module("mtt-gpu-solver_b200.preflop")
    allin = pf.allin_matrix(pf.REFERENCE)
    mats = pf.flop_class_matrices(np.ascontiguousarray(mtt.canonical_flops()[::170, :3]), pf.REFERENCE)
    w = np.linspace(0.5, 1.5, mats.shape[0]).astype(np.float32)
    torch.cuda.synchronize()
    want = [t.cpu() for t in pf.dcfr(w, mats, allin, iters=400)]
    side = torch.cuda.Stream()
    with torch.cuda.stream(side):
        for _ in range(3):
            got = [t.clone() for t in pf.dcfr(w, mats, allin, iters=400)]
            side.synchronize()
            assert all(torch.equal(a, b.cpu()) for a, b in zip(want, got))
