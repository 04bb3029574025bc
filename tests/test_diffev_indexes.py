"""The index tensors of the differentiable EV: finished on the host and copied,
so that no later call on another stream can meet them half made."""
import importlib

import numpy as np
import pytest

SIZES = [(3, 5, 10, 7), (4, 4, 9, 9)]                      # rows0, rows1, hands0, hands1


class _Batch:
    """What StrategyEV reads of a batch, without a device."""

    def __init__(self, sizes):
        rng = np.random.default_rng(0)
        self.n, self.meta = len(sizes), sizes
        self.combos = [tuple(np.sort(rng.choice(1326, h, replace=False)) for h in s[2:]) for s in sizes]

    def layout(self):
        pad = lambda h: (h + 3) // 4 * 4
        rows, rng, tr, tg = [], [], 0, 0
        for r0, r1, h0, h1 in self.meta:
            rows.append((tr, tr + r0 * pad(h0)))
            rng.append(tg)
            tr += r0 * pad(h0) + r1 * pad(h1)
            tg += pad(h0) + pad(h1)
        return {"rows_off": np.array(rows), "range_off": np.array(rng), "total_rows": tr, "total_range": tg}

    def close(self):
        pass


@pytest.mark.parametrize("sizes", [SIZES, SIZES[:1] * 3])
def test_indexes_are_made_on_the_host(monkeypatch, sizes):
    import torch
    from torch.utils._python_dispatch import TorchDispatchMode
    dv = importlib.import_module("mtt-gpu-solver_b200.diffev")
    monkeypatch.setattr(dv, "RiverBatch", lambda subs: _Batch(subs))
    made = []

    class Log(TorchDispatchMode):
        def __torch_dispatch__(self, func, types, args=(), kwargs=None):
            made.append(func.__name__)
            return func(*args, **(kwargs or {}))

    with Log():
        ev = dv.StrategyEV(sizes, device="cpu")
        rows, rng = ev.seg_rows, ev.seg_range
    assert {f for f in made if not f.startswith(("_to_copy", "detach", "alias", "lift_fresh"))} == set()
    lay = ev.batch.layout()
    assert len(rows) == lay["total_rows"] and len(rng) == lay["total_range"]
    assert all(int(rows[o]) == s for s, offs in enumerate(lay["rows_off"]) for o in offs)
    assert all(int(rng[o]) == s for s, o in enumerate(lay["range_off"]))
    r = [torch.rand(ev.n, 1326) for _ in range(2)]
    packed = ev.pack_ranges(*r)
    for s in range(ev.n):
        at = int(lay["range_off"][s])
        for p in range(2):
            c = ev.batch.combos[s][p]
            assert torch.equal(packed[at:at + len(c)], r[p][s, torch.from_numpy(c)])
            at += (len(c) + 3) // 4 * 4


@pytest.mark.gpu
@pytest.mark.parametrize("hands", [(300, 200), (250, 250)])
def test_made_on_one_stream_used_on_another(mtt, wl, cuda, hands):
    import torch
    importlib.import_module("mtt-gpu-solver_b200.diffev")
    subs = [wl.diff_boards(n=1, seed=60 + k, n_hands=h)[0][0] for k, h in enumerate(hands)]
    busy = torch.empty(1 << 28, dtype=torch.uint8, device=cuda)
    r = torch.rand(2, 1326, device=cuda, requires_grad=True)
    w = torch.rand(2, device=cuda)

    def use(ev):
        lg = torch.zeros(ev.total_rows, device=cuda, requires_grad=True)
        packed = ev.pack_ranges(r, r)
        return [packed.detach()] + list(torch.autograd.grad(ev(lg, packed), [lg, r], w))

    want = use(mtt.diffev.StrategyEV(subs))
    torch.cuda.synchronize()
    side = torch.cuda.Stream()
    with torch.cuda.stream(side):
        for _ in range(8):
            busy.fill_(1)                                  # work of the stream that makes the indexes
        ev = mtt.diffev.StrategyEV(subs)
    assert all(torch.equal(a, b) for a, b in zip(want, use(ev)))
