"""The four-hands-a-thread evaluator at its remainders and alignments of
either pointer, with flushes in every position of a group of four."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [4095, 4096, 4097, 4098, 4099, 5120])
@pytest.mark.parametrize("skip_in,skip_out", [(0, 0), (4, 1), (1, 0), (0, 3)])
def test_remainders_and_alignments(mtt, orc, cuda, n, skip_in, skip_out):
    import importlib
    import torch
    lib = importlib.import_module("mtt-gpu-solver_b200._lib").lib()
    rng = np.random.default_rng(n)
    hands = np.stack([rng.choice(52, size=7, replace=False) for _ in range(n)]).astype(np.uint8)
    suited = np.stack([rng.choice(13, size=7, replace=False) for _ in range(n)]).astype(np.uint8) * 4 + 2
    for k in range(n):                                    # every pattern of flushes over groups of four
        if (k // 4 >> (k % 4)) & 1:
            hands[k] = suited[k] if k % 3 else np.r_[suited[k, :5], 0, 1]
    src = torch.zeros(7 * n + skip_in, dtype=torch.uint8, device=cuda)
    src[skip_in:] = torch.from_numpy(hands.reshape(-1)).to(cuda)
    dst = torch.full((n + skip_out + 1,), -7, dtype=torch.int32, device=cuda)
    st = lib.mtt_eval7(ctypes.c_void_p(src.data_ptr() + skip_in), ctypes.c_void_p(dst.data_ptr() + 4 * skip_out), n,
                       ctypes.c_void_p(torch.cuda.current_stream().cuda_stream))
    assert st == 0
    got = dst.cpu().numpy()
    assert np.array_equal(got[skip_out:skip_out + n].view(np.uint32), orc.eval7(hands))
    assert (got[:skip_out] == -7).all() and got[-1] == -7
