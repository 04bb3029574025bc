"""The whole-tree sweeps of small batches against the level kernels, bit for
bit: the same subgames solved in a batch that is too large for them and on
their own, under every update rule, with the exploitability gate, beside a
subgame that deals cards, and at tree sizes of every shared-memory class."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _same(a, b):
    for k in a:
        assert np.array_equal(a[k].view(np.uint8), b[k].view(np.uint8)), k


def _solve(mtt, subs, p, graph, vectors=()):
    b = mtt.RiverBatch(subs)
    b.solve(p, graph=graph)
    out = [b.read(s) for s in range(b.n)]
    for s in vectors:
        out[s]["reach"], out[s]["cfv"] = b.read_vectors(s, len(subs[s]["nodes"]))
    res = b.results() if p.exploitability else np.zeros((b.n, 6))
    it = b.iterations()
    b.close()
    return out, res, it


@pytest.mark.parametrize("algo", [0, 1])
@pytest.mark.parametrize("alternate", [True, False])
@pytest.mark.parametrize("semantics", [0, 1])
def test_small_batches_equal_level_launches(mtt, wl, cuda, algo, alternate, semantics):
    subs = wl.river_batch(n=40, seed=17, min_support=350, max_support=700)      # over 444 slices of 32 hands
    assert sum((max(len(g["combos0"]), len(g["combos1"])) + 31) // 32 for g in subs) > 444
    subs = sorted(subs, key=lambda g: len(g["nodes"]))
    p = mtt.solve_params(iters=7, algo=algo, alternate=alternate, semantics=semantics, avg_power=2.0)
    pick = [0, 13, 26, 39]                                                       # smallest to largest tree
    want, wres, _ = _solve(mtt, subs, p, True, pick)
    for graph in (False, True):
        got, gres, _ = _solve(mtt, [subs[k] for k in pick], p, graph, range(4))
        for n, k in enumerate(pick):
            _same(want[k], got[n])
            assert np.array_equal(wres[k], gres[n])


@pytest.mark.parametrize("alternate", [True, False])
def test_nodes_that_share_rows_equal_level_launches(mtt, wl, cuda, alternate):
    """A caller's tree in which a node uses its ancestor's regret rows: one
    level works on them after the other, in small batches as in large ones."""
    subs = wl.river_batch(n=40, seed=17, min_support=350, max_support=700)
    g = max(subs, key=lambda s: len(s["nodes"]))
    nodes = g["nodes"].copy()
    parent = np.full(len(nodes), -1)
    for i, nd in enumerate(nodes):
        if nd["type"] == 0:
            parent[nd["children_offset"]:nd["children_offset"] + nd["num_actions"]] = i
    shared = 0
    for i, nd in enumerate(nodes):
        a = parent[i]
        while nd["type"] == 0 and a >= 0 and not shared:
            if nodes[a]["player"] == nd["player"] and nodes[a]["num_actions"] >= nd["num_actions"]:
                nodes[i]["infoset_offset"] = nodes[a]["infoset_offset"]
                shared += 1
            a = parent[a]
    assert shared == 1
    g["nodes"] = nodes
    k = next(i for i, s in enumerate(subs) if s is g)
    p = mtt.solve_params(iters=7, alternate=alternate)
    want, _, _ = _solve(mtt, subs, p, True, [k])
    got, _, _ = _solve(mtt, [g], p, True, [0])
    _same(want[k], got[0])


@pytest.mark.parametrize("hands", [1, 3, 31, 33, 128])
def test_slice_edges(mtt, wl, orc, cuda, hands):
    g = wl.river_uniform(seed=hands, n_hands=hands, raise_cap=2)
    (got,), _, _ = _solve(mtt, [g], mtt.solve_params(iters=4, alternate=True), True)
    o = orc.cfr_solve(g, 4, alternate=1)
    for k in ("R0", "R1", "S0", "S1"):
        scale = max(np.abs(o[k]).max(), 1e-30)
        assert np.abs(got[k] - o[k].reshape(got[k].shape)).max() <= 1e-4 * scale


@pytest.mark.parametrize("alternate", [True, False])
def test_gate_and_repeated_solves(mtt, wl, cuda, alternate):
    subs = wl.river_batch(n=6, seed=5, min_support=200, max_support=400, max_sizes=2)
    p = mtt.solve_params(iters=20, alternate=alternate, target_expl=0.004, max_iters=80, chunk_iters=20)
    b = mtt.RiverBatch(subs)
    b.solve(p, graph=True)
    its, first = b.iterations(), [b.read(s) for s in range(b.n)]
    assert its.max() <= 80 and (its.min() < its.max() or not alternate)          # simultaneous updates may all need the limit
    b.solve(mtt.solve_params(iters=3, alternate=alternate), graph=True)          # another run length in between
    b.solve(p, graph=True)
    for s in range(b.n):
        _same(first[s], b.read(s))
    b.close()
    for s, n in enumerate(its):                                                  # each as one run of that length
        (one,), _, _ = _solve(mtt, [subs[s]], mtt.solve_params(iters=int(n), alternate=alternate), False)
        _same(first[s], one)


@pytest.mark.parametrize("alternate", [True, False])
def test_beside_a_turn_subgame(mtt, wl, cuda, alternate):
    turn = wl.turn_dcfr(seed=2, n_hands=60)
    turn["nodes"], turn["rows"], _ = mtt.build_tree(60.0, 90.0, [0.75], raise_cap=1, street=4, board=turn["board"])
    subs = [wl.river_uniform(seed=3, n_hands=150), turn, wl.river_uniform(seed=4, n_hands=90)]
    p = mtt.solve_params(iters=9, algo=1, alternate=alternate)
    both, res, _ = _solve(mtt, subs, p, True, range(3))
    for k in range(3):
        (one,), r, _ = _solve(mtt, [subs[k]], p, True, [0])
        _same(both[k], one)
        assert np.array_equal(res[k], r[0])


@pytest.mark.parametrize("algo", [0, 1])
@pytest.mark.parametrize("semantics", [0, 1])
def test_four_player_small_batches_equal_level_launches(mtt, wl, cuda, algo, semantics):
    """Four-player subgames of one batch past the tree sweeps' limit (2,368
    CTAs of 16 hands of one player) and on their own."""
    import importlib
    mw = importlib.import_module("mtt-gpu-solver_b200.multiway")
    subs = [wl.multiway_icm(seed=4 + k, n_hands=1050 - 11 * k, raise_cap=2) for k in range(13)]
    assert sum(4 * ((len(g["combos"]) + 15) // 16) for g in subs) > 2368
    subs += [wl.multiway_icm(seed=20, n_hands=3, raise_cap=1), wl.multiway_icm(seed=21, n_hands=129, raise_cap=1)]
    p = mtt.solve_params(iters=5, algo=algo, semantics=semantics)

    def solve(gs, graph):
        b = mw.MultiwayBatch(gs)
        b.solve(p, graph=graph)
        out = [b.read(s) for s in range(b.n)]
        v = b.values()
        b.solve(p, graph=graph)                       # again from zero, after the values pass
        for s in range(b.n):
            assert all(np.array_equal(x, y) for x, y in zip(out[s]["R"], b.read(s)["R"]))
        b.close()
        return out, v

    many, mv = solve(subs, True)
    for k in (0, 12, 13, 14):
        for graph in (False, True):
            (one,), v = solve([subs[k]], graph)
            for q in range(4):
                assert np.array_equal(many[k]["R"][q].view(np.uint32), one["R"][q].view(np.uint32))
                assert np.array_equal(many[k]["S"][q].view(np.uint32), one["S"][q].view(np.uint32))
            assert np.array_equal(many[k]["cfv"], one["cfv"]) and np.array_equal(mv[k], v[0])
