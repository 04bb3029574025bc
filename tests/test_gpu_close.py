"""A batch whose root values were read is closed while another batch is being
solved: closing waits for the batch's own work, not for the device."""
import pytest

pytestmark = pytest.mark.gpu


def test_close_does_not_wait_for_other_batches(mtt, wl, cuda):
    import torch
    busy = mtt.RiverBatch(wl.river_batch(n=256, seed=2))
    one = mtt.RiverBatch(wl.river_batch(n=2, seed=3))
    p = mtt.solve_params(iters=300, exploitability=False)
    mine, other = torch.cuda.Stream(), torch.cuda.Stream()
    busy.solve(p, graph=True, stream=other)                # allocations and the graph's capture are behind it
    one.solve(mtt.solve_params(iters=3), stream=mine)
    values = one.root_values(1)
    assert all(v.any() for v in values) and [len(v) for v in values] == [one.meta[1][k] for k in (2, 3, 2, 3)]
    done = torch.cuda.Event()
    busy.solve(p, graph=True, stream=other)                # some 100 ms of work
    done.record(other)
    one.close()
    assert not done.query()
    other.synchronize()
    busy.close()
