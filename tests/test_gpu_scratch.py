"""The calls' scratch memory: after a device reset, inside a captured graph,
and from several streams and threads at once."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

_HANDS = np.array([(a, b) for a in range(52) for b in range(a + 1, 52)], np.uint8)


def _inputs(cuda, seed, H=300):
    import torch
    rng = np.random.default_rng(seed)
    board = rng.choice(52, size=4, replace=False).astype(np.uint8)
    hands = _HANDS[np.sort(rng.choice(1326, size=H, replace=False))]
    return torch.from_numpy(board).to(cuda), torch.from_numpy(hands).to(cuda)


def test_scratch_after_device_reset(cuda, tmp_path):
    import os
    import subprocess
    import sys
    from test_zz_no_alloc import _RESET_SCRIPT
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    head, tail = _RESET_SCRIPT.split("assert rt.cudaDeviceReset() == 0")
    script = tmp_path / "reset_check.py"     # the allocating entry point after the reset
    script.write_text(head + "assert rt.cudaDeviceReset() == 0" + tail.replace("_noalloc", ""))
    r = subprocess.run([sys.executable, str(script), root], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and "reset ok" in r.stdout, r.stdout + r.stderr


def test_scratch_in_a_captured_graph(mtt, cuda):
    import torch
    board, hands = _inputs(cuda, 1)
    want = mtt.board_showdown_counts(board, hands)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        got = mtt.board_showdown_counts(board, hands)
    for t in got:
        t.fill_(-7)
    for _ in range(2):
        graph.replay()
    torch.cuda.synchronize()
    assert all(torch.equal(a, b) for a, b in zip(want, got))


def test_scratch_from_streams_and_threads(mtt, cuda):
    import threading
    import torch
    jobs = [_inputs(cuda, 10 + k, H=200 + 40 * k) for k in range(4)]
    want = [mtt.board_showdown_counts(*j) for j in jobs]
    torch.cuda.synchronize()
    bad = []

    def work(k):
        torch.cuda.set_device(cuda)
        s = torch.cuda.Stream()
        for _ in range(20):
            with torch.cuda.stream(s):
                got = mtt.board_showdown_counts(*jobs[k])
            s.synchronize()
            if not all(torch.equal(a, b) for a, b in zip(want[k], got)):
                bad.append(k)
        mtt.trim_pool()

    th = [threading.Thread(target=work, args=(k,)) for k in range(4)]
    [t.start() for t in th]
    [t.join() for t in th]
    assert not bad
