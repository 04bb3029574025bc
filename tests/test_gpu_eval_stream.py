"""The evaluator given a stream that is not the caller's current one: scores and
inputs are in order with the current stream, without a wait of the caller's."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1024, 200000])
def test_evaluator_given_a_stream(mtt, orc, cuda, n):
    import torch
    rng = np.random.default_rng(n)
    hands = np.argsort(rng.random((n, 52)), axis=1)[:, :7].astype(np.uint8)
    want = orc.eval7(hands)
    cards = torch.from_numpy(hands).to(cuda)
    mine = cards.clone()
    busy = torch.empty(1 << 28, dtype=torch.uint8, device=cuda)
    side = torch.cuda.Stream()
    torch.cuda.synchronize()
    with torch.cuda.stream(side):
        for _ in range(8):
            busy.fill_(1)                                  # the call waits behind this work of its stream
    got = mtt.eval7(mine, stream=side)
    del mine                                               # nothing else keeps the input
    other = torch.zeros_like(cards)
    assert np.array_equal(got.cpu().numpy().view(np.uint32), want)
    assert not other.any()
