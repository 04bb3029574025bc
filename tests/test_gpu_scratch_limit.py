"""The flop matrices where the device has little memory left: the call takes
fewer flops a pass instead of failing, with the same result."""
import importlib

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mode", [0, 1])
def test_flop_matrices_with_little_memory(mtt, cuda, mode):
    import torch
    pf = importlib.import_module("mtt-gpu-solver_b200.preflop")
    flops = np.ascontiguousarray(mtt.canonical_flops()[::70, :3])
    want = pf.flop_class_matrices(flops, mode)
    torch.cuda.synchronize()
    mtt.trim_pool()
    torch.cuda.empty_cache()
    fill = torch.empty(torch.cuda.mem_get_info()[0] - (150 << 20), dtype=torch.uint8, device=cuda)
    try:
        got = pf.flop_class_matrices(flops, mode)
        torch.cuda.synchronize()
    finally:
        del fill
        mtt.trim_pool()
        torch.cuda.empty_cache()
    assert torch.equal(want, got)
