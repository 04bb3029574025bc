"""The flop matrices' correct mode (all 1,326 combos, half ties, the last
villain tile partly empty) against a direct count on the CPU, and a subset
that does not fill one pass, against the oracle."""
import importlib

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture
def pf():
    return importlib.import_module("mtt-gpu-solver_b200.preflop")


def _class_matrix(orc, pf_lib, flop):
    """Mean equity of class pairs over every flop-compatible combo pair: the reference's runout subsample of the
    hero's 47-card deck, ties one half, in double precision."""
    pairs = np.array([(a, b) for a in range(52) for b in range(a + 1, 52)])
    live = [k for k, p in enumerate(pairs) if not set(p) & set(flop)]
    cls = np.array([pf_lib.mtt_pf_combo_class(int(a), int(b)) for a, b in pairs])
    deck = [c for c in range(52) if c not in flop]
    score = {}
    for i, t in enumerate(deck):
        for r in deck[i + 1:]:
            hands = np.array([list(flop) + list(pairs[k]) + [t, r] for k in live], np.uint8)
            score[t, r] = orc.eval7(hands).astype(np.int64)
    pl = pairs[live]
    hit = {c: (pl == c).any(axis=1) for c in deck}
    tot, cnt = np.zeros((169, 169)), np.zeros((169, 169))
    for n, h in enumerate(live):
        own = [c for c in deck if c not in pairs[h]]
        num, den = np.zeros(len(live)), np.zeros(len(live))
        for i in range(0, 47, 2):
            for j in range(i + 1, 47, 3):
                s = score[own[i], own[j]]
                ok = ~(hit[own[i]] | hit[own[j]])
                num += ok * ((s[n] > s) + 0.5 * (s[n] == s))
                den += ok
        ok = (den > 0) & ~(hit[pairs[h][0]] | hit[pairs[h][1]])
        eq = np.where(ok, num / np.maximum(den, 1), 0.0)
        m = eq > 0
        np.add.at(tot[cls[h]], cls[live][m], eq[m])
        np.add.at(cnt[cls[h]], cls[live][m], 1.0)
    return np.where(cnt > 0, tot / np.maximum(cnt, 1), 0.5).T


def test_correct_mode_flop_matrix(pf, orc, cuda):
    flop = np.array([[3, 24, 50]], np.uint8)
    got = pf.flop_class_matrices(flop, pf.CORRECT).cpu().numpy()[0]
    want = _class_matrix(orc, pf.lib(), [3, 24, 50])
    # a class mean of at most 144 equities in float32: 144 roundings of sums up to 144, then one division
    assert np.abs(got - want).max() <= 145 * 2.0 ** -24


@pytest.mark.parametrize("n", [1, 2, 23, 24])
def test_pass_boundaries(pf, orc, cuda, n):
    flops = np.ascontiguousarray(orc.gen_flops()[::71][:n, :3]) if n > 2 else np.array([[0, 1, 2], [8, 21, 51]], np.uint8)[:n]
    assert len(flops) == n
    got = pf.flop_class_matrices(flops, pf.REFERENCE).cpu().numpy()
    for k in sorted({0, n - 1}):
        want = orc.pf_flop_class(flops[k])
        assert np.array_equal(got[k].view(np.uint32), np.asarray(want, np.float32).reshape(169, 169).view(np.uint32))
