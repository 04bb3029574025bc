"""The differentiable EV's equal-length scaling and flat gathers against the
indexed forms they stand in for, over even and uneven subgames, other range
widths, strides and types, second derivatives and batched gradients."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _ev(mtt, wl, sizes):
    subs = []
    for k, h in enumerate(sizes):
        subs += wl.diff_boards(n=1, seed=50 + k, n_hands=h)[0]
    return mtt.diffev.StrategyEV(subs)


def _indexed(ev, r0, r1):
    import torch
    out = torch.zeros(ev.total_range, device=ev.device)
    for p, r in enumerate((r0, r1)):
        out = out.index_put((ev._ridx[p],), r[ev._rsub[p], ev._rcmb[p]].float())
    return out


@pytest.fixture
def dv(mtt):
    import importlib
    importlib.import_module("mtt-gpu-solver_b200.diffev")
    return mtt


@pytest.mark.parametrize("sizes", [(37, 37, 37), (40,), (21, 64, 33)])
@pytest.mark.parametrize("form", ["plain", "wide", "transposed", "double", "more_rows"])
def test_forms_agree(dv, wl, cuda, sizes, form):
    import torch
    ev = _ev(dv, wl, sizes)
    n, g = ev.n, torch.Generator(device="cuda").manual_seed(1)
    logits = torch.randn(ev.total_rows, device="cuda", generator=g)
    shape = {"wide": (n, 1400), "transposed": (1326, n), "more_rows": (n + 2, 1326)}.get(form, (n, 1326))
    base = [torch.rand(shape, device="cuda", generator=g, dtype=torch.float64 if form == "double" else torch.float32)
            for _ in range(2)]
    w = torch.rand(n, device="cuda", generator=g)
    got = []
    for indexed in (False, True):
        lg = logits.clone().requires_grad_()
        rs = [(b.t() if form == "transposed" else b).detach().requires_grad_() for b in base]
        packed = _indexed(ev, *rs) if indexed else ev.pack_ranges(*rs)
        v = ev(lg, packed)
        if indexed:                                  # the gradients as products by an index per element
            _, g_r, g_l = ev.batch.ev_grad(lg.detach(), packed.detach())
            grads = [g_l * w[ev.seg_rows]] + list(torch.autograd.grad(packed, rs, g_r * w[ev.seg_range]))
        else:
            grads = list(torch.autograd.grad(v, [lg] + rs, w))
        got.append([packed.detach(), v.detach()] + grads)
    assert all(torch.equal(a, b) for a, b in zip(*got))
    ev.close()


@pytest.mark.parametrize("sizes", [(37, 37), (21, 64)])
def test_second_derivative_and_batched_gradients(dv, wl, cuda, sizes):
    import torch
    ev = _ev(dv, wl, sizes)
    lg = torch.randn(ev.total_rows, device="cuda").requires_grad_()
    r = torch.rand(ev.n, 1326, device="cuda").requires_grad_()
    packed = ev.pack_ranges(r, r)
    v = ev(lg, packed)
    w = torch.rand(ev.n, device="cuda").requires_grad_()
    (gl,) = torch.autograd.grad(v, lg, w, create_graph=True)
    (gw,) = torch.autograd.grad(gl.sum(), w, retain_graph=True)
    _, _, g_l = ev.batch.ev_grad(lg.detach(), packed.detach())
    want = torch.zeros(ev.n, device="cuda", dtype=torch.float64).index_add_(0, ev.seg_rows, g_l.double())
    # a sum of m float32 terms: m roundings of at most 2^-24 of the terms' absolute sum
    mag = torch.zeros(ev.n, device="cuda", dtype=torch.float64).index_add_(0, ev.seg_rows, g_l.double().abs())
    assert ((gw.double() - want).abs() <= ev.total_rows * 2.0 ** -24 * mag).all()
    eye = torch.eye(ev.n, device="cuda")
    many = torch.autograd.grad(v, [lg, r], eye, is_grads_batched=True, retain_graph=True)
    for k in range(ev.n):
        one = torch.autograd.grad(v, [lg, r], eye[k], retain_graph=True)
        assert all(torch.equal(m[k], o) for m, o in zip(many, one))
    ev.close()
