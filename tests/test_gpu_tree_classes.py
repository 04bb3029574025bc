"""The whole-tree sweeps at the slice widths that the largest and the smallest
trees take (heads-up: 8 hands in the class of one CTA an SM; four players: 4
and 32 hands), and trees past the limit, which take the level launches: bit
for bit the same as in a batch that takes the level launches."""
import importlib

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

KB = 1024


def _smem(g, lg, sim):
    """Bytes of a slice of 4 << lg hands, the most of any player: without its level bounds, and with one per node
    (what decides whether a tree takes these sweeps at all)."""
    nodes, low, high = g["nodes"], 0, 0
    dec = int((nodes["type"] == 0).sum())
    term = len(nodes) - dec
    for q, rows in enumerate(g["rows"]):
        own = int(((nodes["type"] == 0) & (nodes["player"] == q)).sum())
        slots = rows + (max(2 * rows + 1, term) if sim else 2 * rows + 1 + term)
        ints = own + term + (len(nodes) + 1) // 2
        low = max(low, (slots << lg) * 16 + dec * 16 + ints * 4)
        high = max(high, (slots << lg) * 16 + dec * 16 + (ints + 2 * (dec + 1) + 3) // 4 * 16)
    return low, high


def _heads_up(mtt, wl, spr, n_hands, seed):
    g = wl.river_uniform(seed=seed, n_hands=n_hands)
    g["nodes"], g["rows"], _ = mtt.build_tree(100.0, 100.0 * spr, [0.25, 0.5, 0.8, 1.2, 1.8], raise_cap=3)
    return g


@pytest.mark.parametrize("alternate", [True, False])
@pytest.mark.parametrize("n_hands", [33, 64])
def test_heads_up_classes(mtt, wl, cuda, alternate, n_hands):
    one, past = _heads_up(mtt, wl, 12.0, n_hands, 5), _heads_up(mtt, wl, 20.0, n_hands, 6)
    assert _smem(one, 1, False)[0] > 110 * KB and _smem(one, 1, False)[1] <= 224 * KB and _smem(past, 1, False)[1] > 224 * KB
    p = mtt.solve_params(iters=6, alternate=alternate)

    def solve(subs, k):
        b = mtt.RiverBatch(subs)
        b.solve(p)
        r = b.read(k)
        r["reach"], r["cfv"] = b.read_vectors(k, len(subs[k]["nodes"]))
        res = b.results()[k]
        b.close()
        return r, res

    fill = wl.river_batch(n=40, seed=17, min_support=350, max_support=700)       # over three slices of 32 hands an SM
    for g in (one, past):
        (want, wres), (got, gres) = solve([g] + fill, 0), solve([g], 0)
        assert all(np.array_equal(want[k], got[k]) for k in want)
        assert np.array_equal(wres, gres)


@pytest.mark.parametrize("algo", [0, 1])
def test_four_player_slices(mtt, wl, cuda, algo):
    mw = importlib.import_module("mtt-gpu-solver_b200.multiway")

    def sub(stack, cap, n_hands, seed):
        g = wl.multiway_icm(seed=seed, n_hands=n_hands, raise_cap=1)
        g["nodes"], g["rows"], _ = mw.build_tree(4.0, [stack] * 4, [0.5, 1.0], 1.0, cap)
        return g

    narrow, wide = [sub(40.0, 3, 41, 4)], [sub(20.0, 1, 1050, 5), sub(20.0, 1, 1043, 6)]
    past = sub(100.0, 3, 3, 7)
    assert _smem(narrow[0], 1, True)[0] > 112 * KB and _smem(narrow[0], 0, True)[1] <= 224 * KB
    # slices of 8 hands make 528 CTAs a subgame and slices of 16 264, so two take 32 (one wave is 296)
    assert all(_smem(g, 3, True)[1] <= 112 * KB for g in wide) and _smem(past, 0, True)[1] > 224 * KB
    p = mtt.solve_params(iters=4, algo=algo)

    def solve(subs):
        b = mw.MultiwayBatch(subs)
        b.solve(p, graph=True)
        out = [b.read(s) for s in range(b.n)]
        v = b.values()
        b.close()
        return out, v

    for subs in (narrow, wide):
        (got, gv), (want, wv) = solve(subs), solve(subs + [past])                # one tree past the limit: level launches
        for s in range(len(subs)):
            for k in ("R", "S"):
                assert all(np.array_equal(a, b) for a, b in zip(got[s][k], want[s][k]))
            assert np.array_equal(got[s]["cfv"], want[s]["cfv"]) and np.array_equal(gv[s], wv[s])
