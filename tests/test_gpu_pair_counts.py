"""Packed pair counts at the edges of their tiles, stores and completion
words, against the oracle's integer counts."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

_HANDS = np.array([(a, b) for a in range(52) for b in range(a + 1, 52)], np.uint8)


@pytest.mark.parametrize("nboard", [3, 4, 5])
@pytest.mark.parametrize("H", [2, 4, 63, 64, 65, 68, 130])
def test_counts_at_tile_edges(mtt, orc, cuda, nboard, H):
    import torch
    rng = np.random.default_rng(100 * nboard + H)
    board = rng.choice(52, size=nboard, replace=False).astype(np.uint8)
    hands = _HANDS[np.sort(rng.choice(1326, size=H, replace=False))]     # some touch the board
    got = mtt.board_showdown_counts(torch.from_numpy(board).to(cuda), torch.from_numpy(hands).to(cuda))
    for g, o in zip(got, orc.board_counts(board, hands)):
        assert np.array_equal(g.cpu().numpy(), o)
