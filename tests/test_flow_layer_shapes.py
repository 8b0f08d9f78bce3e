"""The fused coupling layers against a float64 restatement with autograd, at
the edges of their block layout: one configuration and partly filled blocks,
the smallest and largest lattices, one to eight mixture terms (five groups of
outputs need two goes), hidden widths that are not a multiple of eight, both
directions and every stripe offset, forward and inverse.

Tolerances: a pre-activation or parameter sums at most 306 products in FP32
(relative error about 306 * 2^-24 = 2e-5 of the terms' size), the transform's
derivatives amplify it by a few: 2e-4 of the 2-norm.  Where a pre-activation is
within FP32 rounding of the LeakyReLU's kink (18 products: 3e-7) its slope is not
determined; the gradients must then agree with one choice of those slopes.
"""
import itertools
import math

import pytest
import torch
import torch.nn.functional as F

pytestmark = pytest.mark.gpu

TWO_PI = 2 * math.pi


def _reference(th, mu, off, K, w, inverse, flips=()):
    """(theta, logdet, undecided units); flips: units whose slope is taken from the other side."""
    L = th.shape[-1]
    P = th[:, 0] + torch.roll(th[:, 1], -1, -1) - torch.roll(th[:, 0], -1, -2) - th[:, 1]
    r = torch.arange(L, device=th.device)
    rel = (r - off) % 4
    frozen = (rel == 1) | (rel == 2)
    frozen = frozen[:, None].expand(L, L) if mu == 0 else frozen[None, :].expand(L, L)
    ctx = torch.stack([torch.cos(P), torch.sin(P)], 1) * frozen
    pre = F.conv2d(F.pad(ctx, (1,) * 4, mode="circular"), w[0], w[1])
    positive = pre.detach() > 0
    for f in flips:
        positive[f] = ~positive[f]
    h = torch.where(positive, pre, 0.01 * pre)
    prm = F.conv2d(F.pad(h, (1,) * 4, mode="circular"), w[2], w[3])
    links = torch.nonzero(rel == 0).flatten()  # rows (mu = 0) or columns of updated links
    act = links if mu == 0 else (links - 1) % L
    prm, Pa = (prm[:, :, act], P[:, act]) if mu == 0 else (prm[:, :, :, act], P[:, :, act])
    al, wt, shift = torch.exp(prm[:, :K].clamp(-8, 8)), torch.softmax(prm[:, K:2 * K], 1), prm[:, 2 * K]

    def mix(x):
        s, c = torch.sin(x / 2)[:, None], torch.cos(x / 2)[:, None]
        return (wt * 2 * torch.atan2(al * s, c)).sum(1), (wt * al / (c * c + al * al * s * s)).sum(1)

    def wrap(x):
        return x - TWO_PI * torch.round(x.detach() / TWO_PI)

    if inverse:
        z = wrap(Pa - shift)
        with torch.no_grad():
            lo, hi = torch.full_like(z, -math.pi), torch.full_like(z, math.pi)
            for _ in range(60):
                mid = (lo + hi) / 2
                below = mix(mid)[0] < z
                lo, hi = torch.where(below, mid, lo), torch.where(below, hi, mid)
        H, Hp = mix(lo)
        x = lo - (H - z) / Hp.detach()
        delta, logd = x - z - shift, torch.log(mix(x)[1])
    else:
        xc = wrap(Pa)
        H, Hp = mix(xc)
        delta, logd = H + shift - xc, torch.log(Hp)
    full = torch.zeros_like(P)
    full = full.index_copy(1 if mu == 0 else 2, links, delta)
    out = torch.stack([th[:, 0] + full, th[:, 1]] if mu == 0 else [th[:, 0], th[:, 1] + full], 1)
    return out, logd.flatten(1).sum(1), [tuple(i) for i in torch.nonzero(pre.detach().abs() < 3e-7).tolist()]


@pytest.mark.parametrize("L,K,hidden,batch", [
    (4, 1, 4, 1), (4, 8, 12, 131), (8, 2, 20, 3), (12, 7, 8, 150), (16, 6, 32, 300), (20, 3, 28, 5), (28, 5, 16, 2),
    (32, 8, 32, 2), (32, 6, 4, 149)])
@pytest.mark.parametrize("inverse", [False, True])
@pytest.mark.parametrize("mu", [0, 1])
def test_layer_matches_float64(L, K, hidden, batch, inverse, mu):
    from latticeu1_b200.flow import Coupling
    off = (L // 4 + K + mu) % 4
    torch.manual_seed(L + K)
    layer = Coupling(L, mu, off, K, hidden).cuda()
    with torch.no_grad():
        for p in layer.net.parameters():
            p.normal_(0, 0.2)
    th = (torch.rand(batch, 2, L, L, device="cuda") * TWO_PI).requires_grad_()
    g_out, g_ld = torch.randn_like(th), torch.randn(batch, device="cuda")
    wrt = [th] + list(layer.net.parameters())
    out, ld = (layer.inverse_fused if inverse else layer.forward_fused)(th)
    got = [out, ld] + list(torch.autograd.grad([out, ld], wrt, [g_out, g_ld]))
    w64 = [p.detach().bfloat16().double().requires_grad_() for p in layer.net.parameters()]
    th64 = th.detach().double().requires_grad_()
    undecided = _reference(th64, mu, off, K, w64, inverse)[2]
    assert len(undecided) <= 6
    worst = None
    for n in range(len(undecided) + 1):
        for flips in itertools.combinations(undecided, n):
            out64, ld64, _ = _reference(th64, mu, off, K, w64, inverse, flips)
            ref = [out64, ld64] + list(torch.autograd.grad([out64, ld64], [th64] + w64, [g_out.double(), g_ld.double()]))
            err = {k: float((a.detach().double() - b.detach()).norm() / b.detach().norm()) for k, a, b in
                   zip(("theta", "logdet", "d theta", "dW1", "dB1", "dW2", "dB2"), got, ref)}
            if worst is None or max(err.values()) < max(worst.values()):
                worst = err
    assert max(worst.values()) < 2e-4, (worst, len(undecided))
