"""A turn subgame that is one depth-limit leaf, beside river subgames small
enough for the whole-tree sweeps: its root values are those it has alone."""
import importlib

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _leaf_root(mtt):
    dl = importlib.import_module("mtt-gpu-solver_b200.depthlimit")
    g = dl.subgame(dl.turn_spot(seed=3), True)
    leaf = g["nodes"][g["nodes"]["type"] == mtt.NODE_LEAF][:1].copy()
    leaf["depth"] = 0
    g["nodes"], g["rows"] = leaf, (0, 0)
    return g


def _values(mtt, subs, k, p, graph):
    b = mtt.RiverBatch(subs)
    b.set_leafnet(None)
    b.solve(p, graph=graph)
    r = b.read(k)
    b.close()
    return r["cfv0"], r["cfv1"]


@pytest.mark.parametrize("alternate", [True, False])
@pytest.mark.parametrize("graph", [True, False])
def test_leaf_root_beside_small_rivers(mtt, wl, cuda, alternate, graph):
    g = _leaf_root(mtt)
    p = mtt.solve_params(iters=3, alternate=alternate, exploitability=False)
    want = _values(mtt, [g], 0, p, graph)
    assert all(np.abs(w).max() > 0.0 for w in want)
    got = _values(mtt, [wl.river_uniform(seed=1, n_hands=60), g], 1, p, graph)
    assert all(np.array_equal(w, v) for w, v in zip(want, got))
