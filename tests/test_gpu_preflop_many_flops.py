"""Preflop iterations over more flops than one staging of 128: at its edges
and over several, against the oracle bit for bit."""
import importlib

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nf", [127, 128, 129, 256, 300])
def test_flops_past_one_staging(orc, cuda, nf):
    import torch
    pf = importlib.import_module("mtt-gpu-solver_b200.preflop")
    rng = np.random.default_rng(nf)
    mats = rng.random((nf, 169, 169)).astype(np.float32)
    allin = rng.random((169, 169)).astype(np.float32)
    w = rng.random(nf).astype(np.float32)
    sums, sig = pf.dcfr(w, torch.from_numpy(mats).to(cuda), torch.from_numpy(allin).to(cuda), iters=12)
    torch.cuda.synchronize()
    o_sums, o_sig = orc.pf_dcfr(w, mats, allin, iters=12)
    assert np.array_equal(sums.cpu().numpy()[:, :169], o_sums[:, :169])
    assert np.array_equal(sig.cpu().numpy()[:, :169], o_sig[:, :169])
