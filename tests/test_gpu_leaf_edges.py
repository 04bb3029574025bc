"""The split reduction at row ends, strides and workspace alignments, and the
Adam step's padding, against plain sums."""
import importlib

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("M,N", [(1, 1), (3, 130), (48, 513), (240, 1024), (129, 2652)])
@pytest.mark.parametrize("ldc_extra,ws_skip", [(0, 0), (1, 0), (4, 1), (3, 2)])
@pytest.mark.parametrize("bf16", [False, True])
def test_split_reduction_edges(mtt, cuda, M, N, ldc_extra, ws_skip, bf16):
    import torch
    g = torch.Generator(device="cuda").manual_seed(M + N)
    K = 1024
    A = torch.randn(M, K, device="cuda", generator=g).to(torch.bfloat16)
    B = torch.randn(N, K, device="cuda", generator=g).to(torch.bfloat16)
    bias = torch.randn(N, device="cuda", generator=g)
    mask = (torch.rand(M, N + ldc_extra, device="cuda", generator=g) - 0.3).to(torch.bfloat16)
    buf = torch.full((M, N + ldc_extra), 7.0, device="cuda", dtype=torch.bfloat16 if bf16 else torch.float32)
    ws = torch.empty(16 * M * (N + 4) + 8, device="cuda")[ws_skip:]
    out = buf[:, :N]
    mtt.gemm_bf16(A, B, bias=bias, relu=True, out_bf16=bf16, mask=mask[:, :N], out=out, workspace=ws)
    want = torch.relu(A.double() @ B.double().T + bias.double()) * (mask[:, :N].float() > 0)
    # 1,024 products of magnitude up to 25, float32 sums: 1,024 * 2^-24 of the absolute sum, and one output rounding
    tol = 1e-3 + (2.0 ** -8 if bf16 else 0.0) * want.abs().max().item()
    assert (out.double() - want).abs().max().item() <= tol
    assert bool((buf[:, N:] == 7.0).all())


def test_adam_step_keeps_padding_zero_and_matches_fp64(mtt, cuda):
    import torch
    ln = importlib.import_module("mtt-gpu-solver_b200.leafnet")
    net = ln.LeafNet(batch_cap=64, seed=3)
    g = torch.Generator(device="cuda").manual_seed(1)
    x = torch.randn(64, ln.IN, device="cuda", generator=g)
    t = torch.randn(64, ln.OUT, device="cuda", generator=g)
    before = [net.params(k) for k in range(4)]
    net.train_step(x, t, lr=1e-3)
    for k in range(4):
        p = net.params(k)
        for w, grad, name in (("w", "gw", "weights"), ("b", "gb", "biases")):
            gr = p[grad].astype(np.float64)
            # the first step with the decay constants and their complements in float32, the corrections from double
            f = np.float32
            m, v = float(f(1) - f(0.9)) * gr / float(f(1.0 - 0.9)), float(f(1) - f(0.999)) * gr * gr / float(f(1.0 - 0.999))
            step = float(f(1e-3)) * m / (np.sqrt(v) + float(f(1e-8)))
            live = np.ones(gr.shape, bool)
            if k == 3:
                live[ln.OUT:] = False
            if k == 0 and w == "w":
                live[:, ln.IN:] = False
            want = np.where(live, before[k][w] - step, 0.0)
            # float32 moments (4 roundings each), their quotient and the weight's own rounding
            assert np.abs(p[w] - want).max() <= 1e-3 * 16 * 2.0 ** -24 + 2.0 ** -24 * max(np.abs(want).max(), 1e-3) + 1e-9, name
            assert not p[w][~live].any()
    net.close()
