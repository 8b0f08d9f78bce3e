"""The inverse of the mixture transform in the fused coupling layers.

On the CPU the header itself, compiled for the host: every solution against a
64-bit bisection, over mild and steep mixtures, all numbers of terms, angles
near 0 and near the ends, with the evaluations counted.  On the GPU the same
through the layer and its backward.

Tolerances.  A computed H = sum_k w_k g_k differs from the exact one by at most
2.4e-6 (g up to pi: 3 ulp of the arctangent, 2 + 2 of sine and cosine, 1.3e-6;
8 products and sums, 1.1e-6), so an FP32 solution lies where the exact H is
within 2.4e-6 of z, or on a float next to such a point.
"""
import ctypes
import math
import shutil
import subprocess
from pathlib import Path

import numpy as np
import pytest

ROOT = Path(__file__).resolve().parents[1]
NOISE = 2.4e-6

HOST = r"""
#include <cmath>
static int evals;
static inline float counted(float a, float b) { ++evals; return atan2f(a, b); }
#define atan2f counted
#include "u1_ncp.cuh"
#undef atan2f
using namespace u1b;
template <int K> static double H64(double x, const NcpMix<K> &m) {
  double v = 0;
  for (int k = 0; k < K; ++k) v += m.w[k] * 2.0 * atan2(m.al[k] * sin(0.5 * x), cos(0.5 * x));
  return v;
}
// x: the solver's, xb: 40 FP32 halvings, xe: 64-bit; n: evaluations; off: |H(x) - z| / noise after a step of one ulp
template <int K> static void solve(int n, const float *prm, const float *z, double *out) {
  for (int i = 0; i < n; ++i) {
    float p[2 * K + 1];
    for (int k = 0; k < 2 * K + 1; ++k) p[k] = prm[i * (2 * K + 1) + k];
    NcpMix<K> m;
    ncp_mix<K>(p, m);
    evals = 0;
    const float x = ncp_solve<K>(z[i], m);
    const int used = evals / K;
    float lo = -3.14159265358979f, hi = 3.14159265358979f, g[K], gp[K], s, c, H, Hp;
    for (int it = 0; it < 40; ++it) {
      const float mid = 0.5f * (lo + hi);
      ncp_values<K>(mid, m, H, Hp, g, gp, s, c);
      (H < z[i] ? lo : hi) = mid;
    }
    double a = -M_PI, b = M_PI;
    for (int it = 0; it < 70; ++it) {
      const double mid = 0.5 * (a + b);
      (H64<K>(mid, m) < z[i] ? a : b) = mid;
    }
    // exact H one float below and above the solution
    const double h0 = H64<K>(nextafterf(x, -4.f), m), h1 = H64<K>(nextafterf(x, 4.f), m);
    double *o = out + 5 * i;
    o[0] = x;
    o[1] = 0.5f * (lo + hi);
    o[2] = 0.5 * (a + b);
    o[3] = used;
    o[4] = std::fmax(0.0, std::fmax(h0 - z[i], z[i] - h1));
  }
}
extern "C" void ncp_solutions(int K, int n, const float *prm, const float *z, double *out) {
  switch (K) {
    case 1: return solve<1>(n, prm, z, out);
    case 2: return solve<2>(n, prm, z, out);
    case 3: return solve<3>(n, prm, z, out);
    case 6: return solve<6>(n, prm, z, out);
    default: return solve<8>(n, prm, z, out);
  }
}
"""


@pytest.fixture(scope="module")
def host(tmp_path_factory):
    gxx = shutil.which("g++")
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    include = Path(nvcc).resolve().parents[1] / "include"
    if gxx is None or not (include / "cuda_runtime.h").exists():
        pytest.skip("g++ and the CUDA headers are needed")
    d = tmp_path_factory.mktemp("ncp")
    (d / "h.cpp").write_text(HOST)
    subprocess.run([gxx, "-O2", "-ffp-contract=off", "-w", "-shared", "-fPIC", f"-I{include}",
                    f"-I{ROOT / 'latticeu1_b200' / 'csrc'}", str(d / "h.cpp"), "-o", str(d / "h.so")], check=True)
    return ctypes.CDLL(str(d / "h.so"))


def _terms(rng, n, K, spread):
    """(n, 2K + 1) parameters; spread: standard deviation of log alpha, "all" of [-8, 8], or "ends" of it."""
    p = np.zeros((n, 2 * K + 1), np.float32)
    p[:, :K] = (rng.uniform(-8, 8, (n, K)) if spread == "all" else rng.choice((-8.0, 8.0), (n, K))
                if spread == "ends" else spread * rng.standard_normal((n, K)))
    p[:, K:2 * K] = rng.standard_normal((n, K)) * (2.0 if isinstance(spread, str) else 0.5)
    return p


def _angles(rng, n):
    z = rng.uniform(-math.pi, math.pi, n)
    z[::16] *= 1e-4
    z[1::16] = np.copysign(math.pi - np.abs(z[1::16]) * 1e-6, z[1::16])
    z[2], z[3], z[4] = 0.0, np.float32(math.pi), -np.float32(math.pi)
    return z.astype(np.float32)


@pytest.mark.parametrize("K,spread", [(6, 0.05), (6, 0.3), (6, 1.0), (6, 2.0), (6, 3.0), (6, "all"), (6, "ends"),
                                      (1, "all"), (2, "ends"), (3, 2.0), (8, 1.0), (8, "all"), (8, "ends")])
def test_host_solutions(host, K, spread):
    n = 19200
    rng = np.random.default_rng(K)
    p, z, out = _terms(rng, n, K, spread), _angles(rng, n), np.zeros((n, 5))
    host.ncp_solutions(K, n, p.ctypes.data_as(ctypes.c_void_p), z.ctypes.data_as(ctypes.c_void_p),
                       out.ctypes.data_as(ctypes.c_void_p))
    x, xb, exact, evals, off = out.T
    assert np.all(np.abs(x) <= np.float32(math.pi))
    assert off.max() <= NOISE
    assert np.abs(x - exact).max() <= np.abs(xb - exact).max()
    assert evals.max() <= 40  # never more than the bisection
    longest = evals.reshape(-1, 32).max(1).mean()
    assert longest <= {0.05: 4, 0.3: 5, 1.0: 8, 2.0: 12, 3.0: 17}.get(spread, 30), longest


def _mix64(x, al, w):
    import torch
    s, c = torch.sin(x / 2)[..., None], torch.cos(x / 2)[..., None]
    den = c * c + al * al * s * s
    return ((w * 2 * torch.atan2(al * s, c)).sum(-1), (w * al / den).sum(-1),
            (w * (-al * s * c * (al * al - 1)) / (den * den)).sum(-1))


@pytest.mark.gpu
@pytest.mark.parametrize("mu", [0, 1])
@pytest.mark.parametrize("spread", [0.3, 2.0, 3.0, "all", "ends"])
def test_layer_inverse_and_backward(spread, mu):
    """Every plaquette of a 32^2 layer, batch 1024: the second convolution's weights are zero, so its bias is the
    parameters of all plaquettes and the angles alone vary."""
    import torch

    from latticeu1_b200.flow import Coupling, plaquettes_no
    L, K, batch, off = 32, 6, 1024, 2
    rng = np.random.default_rng(17)
    layer = Coupling(L, mu, off, K, 8).cuda()
    for trial in range(4):
        prm = torch.tensor(_terms(rng, 1, K, spread)[0]).bfloat16()
        prm[2 * K] = 0.3
        with torch.no_grad():
            layer.net[2].bias.copy_(prm.float())
        torch.manual_seed(trial)
        th = (torch.rand(batch, 2, L, L, device="cuda") * (2 * math.pi)).requires_grad_()
        out, ld = layer.inverse_fused(th)
        g_out = torch.randn_like(th)
        g_th, = torch.autograd.grad(out, th, g_out)
        prm = prm.float().cuda()
        al = torch.exp(prm[:K].clamp(-8, 8)).double()  # the kernel's own FP32 terms, to the last rounding
        w = torch.softmax(prm[K:2 * K], 0).double()
        P = plaquettes_no(th.detach()).reshape(batch, -1)[:, layer.act_idx]
        # z = remainder(P - shift) as the kernel rounds it: the difference in FP32, the remainder exact
        d = (P - prm[2 * K]).double()
        two_pi = float(np.float32(2 * math.pi))
        z = d - two_pi * torch.round(d / two_pi)
        delta = (out.detach().double() - th.detach().double())[:, mu].reshape(batch, -1)[:, layer.link_idx]
        x = delta + z + prm[2 * K].double()
        lo, hi = torch.full_like(z, -math.pi), torch.full_like(z, math.pi)
        for _ in range(60):
            mid = (lo + hi) / 2
            below = _mix64(mid, al, w)[0] < z
            lo, hi = torch.where(below, mid, lo), torch.where(below, hi, mid)
        exact = (lo + hi) / 2
        # what the kernel does with x: three roundings at up to 2 pi (xs - z, - shift, theta + change), 2^-22 each,
        # and alpha, w to 3 ulp (they shift z by up to 2 pi 2^-22)
        room = 4 * 2.0 ** -22 * 2
        eps = NOISE + 2 * math.pi * 2.0 ** -22
        low, high = _mix64(x - room, al, w)[0] - z, _mix64(x + room, al, w)[0] - z
        # a steep mixture moves across the whole noise within the rounding of x, a flat one needs the noise in H
        assert float(low.max()) <= eps and float(-high.min()) <= eps, (spread, trial)
        # log det: d log H' / dx is at most alpha / 2 of the steepest term, so compare where the solution fixes it
        H, Hp, dHp = _mix64(exact, al, w)
        dx = eps / Hp + 2.0 ** -22
        safe = ((dHp / Hp).abs() * dx < 1e-2).all(1)
        want = torch.log(Hp).sum(1)
        bound = ((dHp / Hp).abs() * dx * 1.1 + 2.0 ** -18).sum(1)
        assert bool(((ld.double() - want).abs() <= bound + want.abs() * 2.0 ** -23)[safe].all()), (spread, trial)
        # backward with no gradient of the log det: the active plaquettes' gP = gout / H' - gout
        flat = g_out.double().reshape(batch, 2, -1)
        gout = flat[:, mu][:, layer.link_idx]
        gP = torch.zeros(batch, L * L, dtype=torch.float64, device="cuda")
        gP[:, layer.act_idx] = gout / Hp - gout
        gP = gP.reshape(batch, L, L)
        ref = g_out.double() + torch.stack([gP - torch.roll(gP, 1, 1), torch.roll(gP, 1, 2) - gP], 1)
        tol = torch.zeros(batch, L * L, dtype=torch.float64, device="cuda")
        rel = (dHp / Hp).abs() * dx * 1.1 + 2.0 ** -18
        tol[:, layer.act_idx] = torch.where(rel < 1e-2, rel * (gout / Hp).abs() + 2.0 ** -22 * gout.abs(), math.inf)
        tol = tol.reshape(batch, L, L)
        allow = torch.stack([tol + torch.roll(tol, 1, 1), torch.roll(tol, 1, 2) + tol], 1) + 2.0 ** -21 * (
            ref.abs() + g_out.abs().double()) + 2.0 ** -21 * torch.stack([gP.abs() + torch.roll(gP, 1, 1).abs(),
                                                                       torch.roll(gP, 1, 2).abs() + gP.abs()], 1)
        assert bool(((g_th.double() - ref).abs() <= allow).all()), (spread, trial)
