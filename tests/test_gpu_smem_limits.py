"""Batches of different tree sizes solved from two threads at once, each on its
own stream: no solve lowers the shared-memory limit under another's launches."""
import threading

import pytest

pytestmark = pytest.mark.gpu


def test_solves_of_two_tree_sizes_from_two_threads(mtt, wl, cuda):
    import torch
    sizes = []
    for spr, bets, cap in ((12.0, [0.3, 0.6, 1.0, 1.8], 3), (8.0, [0.33, 0.75, 1.5], 3)):
        g = wl.river_uniform(seed=1, n_hands=64)
        g["nodes"], g["rows"], _ = mtt.build_tree(100.0, 100.0 * spr, bets, raise_cap=cap)
        sizes.append((g, len(g["nodes"])))
    assert sizes[0][1] > 2 * sizes[1][1]                   # both above the default limit of 48 KB, by different amounts
    p = mtt.solve_params(iters=40, exploitability=False)
    bad = []

    def work(g):
        torch.cuda.set_device(cuda)
        s = torch.cuda.Stream()
        b = mtt.RiverBatch([g])
        try:
            for _ in range(60):
                b.solve(p, stream=s, graph=False)
        except mtt.MttError as e:
            bad.append(e)
        s.synchronize()
        b.close()

    th = [threading.Thread(target=work, args=(g,)) for g, _ in sizes]
    [t.start() for t in th]
    [t.join() for t in th]
    assert not bad
