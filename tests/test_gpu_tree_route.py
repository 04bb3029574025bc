"""Which batches take the whole-tree sweeps, told by the kernels launched an
iteration (four, or one of each kind and level): those whose slices of one
player are at most about two waves, whatever their trees' size."""
import pytest

pytestmark = pytest.mark.gpu

BETS = [0.25, 0.5, 0.8, 1.2, 1.8]


def _launches(mtt, wl, spr, bets, cap, n, hands):
    nodes, rows, _ = mtt.build_tree(100.0, 100.0 * spr, bets, raise_cap=cap)
    subs = [dict(wl.river_uniform(seed=k, n_hands=hands), nodes=nodes, rows=rows) for k in range(n)]
    b = mtt.RiverBatch(subs)
    counts = []
    for iters in (2, 12):
        at = b.launch_count()
        b.solve(mtt.solve_params(iters=iters, exploitability=False))
        counts.append(b.launch_count() - at)
    b.close()
    return (counts[1] - counts[0]) // 10


@pytest.mark.parametrize("spr,bets,cap,n,hands,tree", [
    (12.0, BETS, 3, 1, 300, True),                  # 2,181 nodes, one CTA an SM: 38 slices of a player
    (12.0, BETS, 3, 10, 300, False),                # 380
    (8.0, [0.3, 0.6, 1.0, 1.8], 3, 4, 1081, True),  # 783 nodes, two CTAs an SM: 544
    (8.0, [0.3, 0.6, 1.0, 1.8], 3, 40, 300, False), # 1,520
    (4.0, [0.5, 1.0], 1, 13, 1081, True),           # 51 nodes: 442
    (4.0, [0.5, 1.0], 1, 14, 1081, False),          # past three slices of 32 hands an SM
])
def test_route(mtt, wl, cuda, spr, bets, cap, n, hands, tree):
    per = _launches(mtt, wl, spr, bets, cap, n, hands)
    assert (per <= 8) if tree else (per > 8)
