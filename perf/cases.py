"""Performance cases: the work users of this package have it do, through its public entry points.

Listed cases (what each stands for is said beside it) and `draw`, which gives
more of the same ranges: lattices from a few thousand links, where launch
latency counts, to half a gigabyte, beyond L2; two, three and four dimensions;
even extents of every residue; single chains, batches, correlators, the
differentiable action and the 2D flow.

A case is a dict of plain values; `prepare` builds what a user's program has
in hand before the call, `run` makes one pass, `work` states the bytes and
operations the pass cannot do without and `exact` gives its result in 64 bits
from plain torch where it has one.  A whole sweep has none: compact U(1)
dynamics is chaotic, so a rounding difference grows to order one within a few
passes and a 64-bit chain is a different chain.
"""
from __future__ import annotations

import math

import numpy as np
import torch
import torch.nn.functional as F

from latticeu1_b200 import Batch, Context, Lattice, Rng
from latticeu1_b200.action import WilsonAction
from latticeu1_b200.flow import Coupling, Flow2D

DEVICE = "cuda:0"

# Lattices of at least this many sites take their measurement from the sweep's
# last pass (Lattice.update_measure); smaller ones are measured by a call of
# its own after the sweep, as the driver program does (its results are then
# summed in one order whatever kernel the tuner picked for the sweep).
FUSED_MIN_SITES = 1 << 19


def listed() -> list[dict]:
    return [
        # The smallest production run: 8^4 from a hot start, delta = pi/2 Metropolis,
        # update and host-side measurement every sweep.  Launch latency.
        _sweep("sweep_8x4", 4, (8, 8, 8, 8), 1.0, window=0.5),
        # The plain chain the 2D flow sampler is judged against.
        _sweep("sweep_2d_32", 2, (32, 0, 0, 32), 6.0),
        # Ragged extents (Nx/2 odd), anisotropic: a lattice no tile divides.
        _sweep("sweep_ragged", 4, (22, 18, 14, 30), 2.0, aniso=2.0),
        # The headline lattice, resident in L2.
        _sweep("sweep_32x4", 4, (32, 32, 32, 32), 1.0),
        # A lattice far beyond L2.
        _sweep("sweep_64x4", 4, (64, 64, 64, 64), 1.0),
        # Configurations that live on the host: in, one measured sweep, out.
        {"name": "host_24x48", "kind": "host", "dims": 4, "nx": 24, "ny": 24, "nz": 24, "nt": 48, "beta": 2.0,
         "aniso": 2.0, "metrop": 1, "ovrn": 4},
        # Many independent chains of uneven volume, measured, configurations recorded.
        {"name": "batch_512", "kind": "batch", "dims": 4, "metrop": 1, "ovrn": 4,
         "chains": "256:16,16,16,16;128:12,12,12,12;128:16,16,16,32"},
        # Two-level Polyakov correlator, multihit on temporal links.
        {"name": "multilevel_24x32", "kind": "multilevel", "nx": 24, "ny": 24, "nz": 24, "nt": 32, "beta": 0.95,
         "n4": 1, "k4": 1, "n2": 20, "k2": 1, "metrop": 1, "ovrn": 4},
        # Single-level measurement of one configuration: plaquettes, Polyakov loop, multihit correlator.
        {"name": "measure_24x32", "kind": "measure", "dims": 4, "nx": 24, "ny": 24, "nz": 24, "nt": 32, "beta": 0.95,
         "aniso": 1.0, "multihit": True},
        # Action and force of a few 4D configurations (forward and backward).
        {"name": "action_16x4", "kind": "action", "dims": 4, "nx": 16, "ny": 16, "nz": 16, "nt": 16, "beta": 1.0,
         "aniso": 1.0, "batch": 8, "dtype": "float32"},
        # One coupling layer of the 32^2 flow, forward and backward at the training batch.
        {"name": "flow_train_32", "kind": "flow_layer", "L": 32, "mu": 0, "off": 1, "K": 6, "hidden": 32,
         "batch": 1024, "inverse": False},
        # Proposals of a whole 8-layer 16^2 flow with their log probabilities.
        {"name": "flow_sample_16", "kind": "flow_sample", "L": 16, "layers": 8, "K": 6, "hidden": 32, "batch": 1024},
    ]


def draw(rng) -> dict:
    kind = rng.choice(("sweep", "sweep", "sweep", "host", "batch", "multilevel", "measure", "action", "flow_layer",
                       "flow_sample"))
    if kind in ("sweep", "host", "measure"):
        dims = rng.choice((2, 3, 4, 4, 4))
        N = _draw_extents(rng, dims, 10, 21 if kind == "sweep" else 19)
        aniso = rng.choice((1.0, 1.0, round(rng.uniform(1.2, 2.5), 3)))
        beta = round(rng.uniform(0.8, 2.0) if dims == 4 else rng.uniform(1.0, 6.0), 3)
        if kind == "measure":
            return {"kind": kind, "dims": dims, **_extents(N), "beta": beta, "aniso": aniso,
                    "multihit": rng.random() < 0.7}
        c = _sweep("", dims, N, beta, aniso, ovrn=rng.choice((1, 2, 3, 4, 4, 5)))
        del c["name"]
        if kind == "host":
            del c["window"], c["hits"]
            c["kind"] = kind
        elif rng.random() < 0.2:
            c["window"], c["hits"] = round(rng.uniform(0.2, 0.9), 3), rng.choice((1, 2, 4))
        return c
    if kind == "batch":
        dims = rng.choice((2, 4, 4))
        parts, left = [], 1 << rng.randint(20, 25)  # links of all chains
        for _ in range(rng.randint(1, 3)):
            N = _draw_extents(rng, dims, 8, 15)
            n = max(1, min(256, left // (3 * dims * _volume(N))))
            parts.append("%d:%d,%d,%d,%d" % ((n,) + N))
        return {"kind": kind, "dims": dims, "chains": ";".join(parts), "metrop": 1, "ovrn": rng.choice((2, 4))}
    if kind == "multilevel":
        N = [2 * rng.randint(3, 10) for _ in range(3)] + [4 * rng.randint(2, 8)]
        return {"kind": kind, **_extents(N), "beta": round(rng.uniform(0.8, 1.1), 3), "n4": rng.randint(1, 2),
                "k4": 1, "n2": rng.randint(3, 12), "k2": rng.randint(1, 2), "metrop": 1, "ovrn": rng.choice((2, 4))}
    if kind == "action":
        dims = rng.choice((2, 3, 4))
        N = _draw_extents(rng, dims, 10, 16)
        most = (1 << 21) // _volume(N)
        return {"kind": kind, "dims": dims, **_extents(N), "beta": round(rng.uniform(0.8, 4.0), 3),
                "aniso": rng.choice((1.0, 1.5)), "batch": max(1, min(1024, int(2 ** rng.uniform(0, math.log2(most))))),
                "dtype": rng.choice(("float32", "float32", "float64"))}
    c = {"kind": kind, "L": 4 * rng.randint(2, 8), "K": rng.randint(2, 8), "hidden": rng.choice((8, 12, 16, 24, 32)),
         "batch": int(2 ** rng.uniform(5, 10))}
    if kind == "flow_layer":
        return {**c, "mu": rng.randint(0, 1), "off": rng.randint(0, 3), "inverse": rng.random() < 0.4}
    return {**c, "layers": rng.choice((4, 8, 16))}


def _sweep(name, dims, N, beta, aniso=1.0, window=0.0, hits=1, metrop=1, ovrn=4) -> dict:
    """window: half-width of the Metropolis proposal over pi (0: the whole circle)."""
    return {"name": name, "kind": "sweep", "dims": dims, **_extents(N), "beta": beta, "aniso": aniso,
            "window": window, "hits": hits, "metrop": metrop, "ovrn": ovrn}


def _extents(N) -> dict:
    return {"nx": int(N[0]), "ny": int(N[1]), "nz": int(N[2]), "nt": int(N[3])}


def _draw_extents(rng, dims, lo, hi) -> tuple:
    """Even extents (Nx, Ny, Nz, Nt), unused ones 0, of a volume about 2^lo..2^hi, log-uniform."""
    target = 2 ** rng.uniform(lo, hi)
    n = []
    for k in range(dims):
        side = target ** (1.0 / (dims - k))
        e = max(4, 2 * round(side * (rng.uniform(0.75, 1.3) if k + 1 < dims else 1.0) / 2))
        n.append(int(e))
        target = max(4.0, target / e)
    return {2: (n[0], 0, 0, n[-1]), 3: (n[0], n[min(1, dims - 1)], 0, n[-1])}.get(dims) or tuple(n)


def _N(case) -> tuple:
    return case["nx"], case["ny"], case["nz"], case["nt"]


def _volume(N) -> int:
    return math.prod(n for n in N if n)


def _chains(case) -> list:
    """(extents, count) of every group of chains."""
    out = []
    for part in case["chains"].split(";"):
        n, ext = part.split(":")
        out.append((tuple(int(x) for x in ext.split(",")), int(n)))
    return out


# --------------------------------------------------------------------- state
class _Buffer:
    """Device memory the library owns, as torch.as_tensor takes it (no copy)."""

    def __init__(self, ptr: int, shape: tuple, typestr: str, owner):
        self.__cuda_array_interface__ = {"data": (ptr, False), "shape": shape, "typestr": typestr, "version": 3}
        self.owner = owner


def _context() -> Context:
    torch.cuda.init()
    return Context(0)


def _generator(seed: int, device=DEVICE) -> torch.Generator:
    g = torch.Generator(device=device)
    g.manual_seed(int(seed))
    return g


def _angles(n: int, seed: int, dtype=torch.float64) -> torch.Tensor:
    """Link angles of a disordered configuration, fluctuating about 0."""
    return (torch.randn(n, generator=_generator(seed), device=DEVICE, dtype=torch.float64) * 0.6).to(dtype)


def _weights(net, seed: int) -> None:
    """Weights of the size a trained layer has, from the seed alone."""
    g = _generator(seed)
    with torch.no_grad():
        for conv, std in ((net[0], 0.25), (net[2], 0.06)):
            for p in (conv.weight, conv.bias):
                p.copy_(torch.randn(p.shape, generator=g, device=DEVICE) * std)


def prepare(case: dict, seed: int) -> dict:
    kind = case["kind"]
    s = {"case": case, "kind": kind}
    if kind in ("sweep", "host", "multilevel", "measure"):
        dims = case.get("dims", 4)
        ctx = _context()
        lat = Lattice(ctx, dims, _N(case), case["beta"], case.get("aniso", 1.0))
        rng = Rng(ctx, 1000 + int(seed))
        s.update(ctx=ctx, lat=lat, rng=rng, obs=torch.zeros(6, dtype=torch.float64, device=DEVICE))
        if kind == "measure":
            lat.import_angles(_angles(lat.nlinks, seed))
            return s
        if case.get("window") or case.get("hits", 1) != 1:
            lat.set_metropolis(case["window"] * math.pi, case["hits"])
        lat.hot_start(rng)
        for _ in range(3):  # towards equilibrium; the first sweep also tunes this geometry's kernels
            lat.update(rng, case["metrop"], case["ovrn"])
        s["links"] = torch.as_tensor(_Buffer(lat.links_ptr(), (lat.nlinks, 2), "<f4", lat), device=DEVICE)
        if kind == "host":
            s["theta"] = torch.empty(lat.nlinks, dtype=torch.float64, pin_memory=True)
            s["out"] = torch.empty(lat.nlinks, dtype=torch.float64, pin_memory=True)
            lat.export_angles(s["theta"])
        lat.synchronize()
    elif kind == "batch":
        ctx = _context()
        beta = np.random.default_rng(int(seed)).uniform(0.8, 1.2, sum(n for _, n in _chains(case)))
        shapes = [N for N, n in _chains(case) for _ in range(n)]
        b = Batch(ctx, [(case["dims"], N, bt) for N, bt in zip(shapes, beta)], seed=1000 + int(seed))
        b.hot_start()
        b.update(case["metrop"], case["ovrn"])
        s.update(ctx=ctx, batch=b, angles=torch.empty(b.total_links, dtype=torch.float64, device=DEVICE))
    elif kind == "action":
        n = case["dims"] * _volume(_N(case))
        th = _angles(case["batch"] * n, seed, getattr(torch, case["dtype"])).reshape(case["batch"], n)
        s.update(action=WilsonAction(case["dims"], _N(case), case["beta"], case["aniso"]), theta=th.requires_grad_(),
                 up=torch.ones(case["batch"], dtype=torch.float64, device=DEVICE))
    elif kind == "flow_layer":
        layer = Coupling(case["L"], case["mu"], case["off"], case["K"], case["hidden"]).to(DEVICE)
        _weights(layer.net, seed)
        s.update(layer=layer, **_flow_inputs(case, seed))
        s["theta"].requires_grad_()
        s["wrt"] = [s["theta"]] + list(layer.net.parameters())
    else:
        flow = Flow2D(case["L"], 2.0, case["layers"], case["K"], case["hidden"]).to(DEVICE)
        for k, layer in enumerate(flow.layers):
            _weights(layer.net, 100 * int(seed) + k)
        s.update(flow=flow, gen=_generator(seed))
    return s


def _flow_inputs(case: dict, seed: int) -> dict:
    g = _generator(int(seed) + 7)
    shape = (case["batch"], 2, case["L"], case["L"])
    return {"theta": torch.rand(shape, generator=g, device=DEVICE) * (2 * math.pi),
            "g_theta": torch.randn(shape, generator=g, device=DEVICE) / case["batch"],
            "g_logdet": torch.full((case["batch"],), -1.0 / case["batch"], device=DEVICE)}


def run(s: dict):
    case, kind = s["case"], s["kind"]
    if kind == "sweep":
        lat = s["lat"]
        if lat.V >= FUSED_MIN_SITES:
            lat.update_measure(s["rng"], case["metrop"], case["ovrn"], s["obs"].data_ptr())
            return {"links": s["links"], "observables": s["obs"]}
        lat.update(s["rng"], case["metrop"], case["ovrn"])
        return {"links": s["links"], "observables": np.array(list(_flat(lat.measure())))}
    if kind == "host":
        lat = s["lat"]
        lat.import_angles_async(s["theta"])
        lat.update(s["rng"], case["metrop"], case["ovrn"])
        lat.measure_async(s["obs"].data_ptr())
        lat.export_angles_async(s["out"])
        lat.synchronize()
        return {"angles": s["out"], "observables": s["obs"]}
    if kind == "batch":
        s["batch"].update(case["metrop"], case["ovrn"], measure=True)
        return {"observables": s["batch"].results_raw(), "angles": s["batch"].export_all(s["angles"])}
    if kind == "multilevel":
        return s["lat"].multilevel(s["rng"], case["n4"], case["k4"], case["n2"], case["k2"], case["metrop"],
                                   case["ovrn"])
    if kind == "measure":
        return {"observables": np.array(list(_flat(s["lat"].measure()))), "correlator": s["lat"].poly_corr(case["multihit"])}
    if kind == "action":
        S = s["action"](s["theta"])
        (force,) = torch.autograd.grad(S, s["theta"], s["up"])
        return {"action": S.detach(), "force": force}
    if kind == "flow_layer":
        layer = s["layer"]
        out, logdet = (layer.inverse_fused if case["inverse"] else layer.forward_fused)(s["theta"])
        grads = torch.autograd.grad([out, logdet], s["wrt"], [s["g_theta"], s["g_logdet"]])
        return {"theta": out.detach(), "logdet": logdet.detach(), "grads": list(grads)}
    th, logq = s["flow"].sample_fused(case["batch"], s["gen"])
    return {"cos": torch.cos(th), "sin": torch.sin(th), "logq": logq}  # the links, as observables take them


def _flat(m: dict):
    for k in ("plaq_ss", "plaq_st", "poly"):
        yield m[k].real
        yield m[k].imag


# ---------------------------------------------------------------------- work
def _update_flops(dims: int) -> int:
    """One link update: 2(d-1) staple terms of two complex products and a sum, and the new link."""
    return 2 * (dims - 1) * 16 + 24


def work(case: dict) -> dict:
    kind = case["kind"]
    if kind in ("sweep", "host", "measure", "multilevel"):
        dims = case.get("dims", 4)
        V = _volume(_N(case))
        n = V * dims
        if kind == "sweep":
            return {"bytes": 16 * n, "flops": n * (case["metrop"] + case["ovrn"]) * _update_flops(dims)}
        if kind == "host":
            return {"bytes": 16 * n, "flops": n * (case["metrop"] + case["ovrn"]) * _update_flops(dims)}
        plaq = V * dims * (dims - 1) // 2
        if kind == "measure":
            return {"bytes": 8 * n, "flops": plaq * 20 + V * (_update_flops(dims) if case["multihit"] else 8)}
        # T2 has (d-1) R Vs (Nt/2) complex doubles, formed from every sub-update
        t2 = 3 * (case["nx"] // 2) * V // 2
        sweeps = case["n4"] * (case["k4"] + case["n2"] * case["k2"]) * (case["metrop"] + case["ovrn"])
        return {"bytes": 8 * n + case["n4"] * 16 * t2,
                "flops": n * sweeps * _update_flops(4) + case["n4"] * case["n2"] * t2 * 8}
    if kind == "batch":
        n = sum(c * case["dims"] * _volume(N) for N, c in _chains(case))
        return {"bytes": 24 * n, "flops": n * (case["metrop"] + case["ovrn"]) * _update_flops(case["dims"])}
    if kind == "action":
        dims, V, size = case["dims"], _volume(_N(case)), 4 if case["dtype"] == "float32" else 8
        return {"bytes": 2 * size * case["batch"] * V * dims, "flops": case["batch"] * V * dims * (dims - 1) * 24}
    L2, K, H = case["L"] ** 2, case["K"], case["hidden"]
    conv = L2 * 18 * H * 2 + L2 // 4 * 9 * H * (2 * K + 1) * 2  # both convolutions of one configuration
    if kind == "flow_layer":
        return {"bytes": case["batch"] * 4 * (2 * L2) * 4, "flops": case["batch"] * 3 * conv}
    return {"bytes": case["batch"] * 4 * 2 * L2 * 2, "flops": case["batch"] * case["layers"] * conv}


# --------------------------------------------------------------------- exact
def exact(case: dict, seed: int):
    kind = case["kind"]
    if kind == "measure":
        return _exact_measure(case, seed)
    if kind == "action":
        return _exact_action(case, seed)
    if kind == "flow_layer":
        return _exact_flow_layer(case, seed)
    if kind == "flow_sample":
        return _exact_flow_sample(case, seed)
    return None


def _natural(theta: torch.Tensor, dims: int, N) -> tuple[torch.Tensor, list]:
    """Angles theta[..., mu*V + parity*V/2 + (lex >> 1)] as [..., mu, x_{d-1}, ..., x_0],
    and the extents x_0..x_{d-1}."""
    ext = {2: [N[0], N[3]], 3: [N[0], N[1], N[3]], 4: list(N)}[dims]
    V = math.prod(ext)
    lex = torch.arange(V, device=theta.device)
    r, par = lex, torch.zeros_like(lex)
    for e in ext:
        par, r = par + r % e, r // e
    where = (lex >> 1) + (par & 1) * (V // 2)
    th = theta.reshape(theta.shape[:-1] + (dims, V))[..., where]
    return th.reshape(th.shape[:-1] + tuple(reversed(ext))), ext


def _at(a: torch.Tensor, mu: int, step: int = 1) -> torch.Tensor:
    """a(x + step mu) of an array indexed [..., x_1, x_0]."""
    return torch.roll(a, -step, dims=-1 - mu)


def _exact_measure(case, seed):
    dims = case["dims"]
    th, ext = _natural(_angles(dims * _volume(_N(case)), seed), dims, _N(case))
    t = dims - 1

    def angle(mu, nu):
        return th[mu] + _at(th[nu], mu) - _at(th[mu], nu) - th[nu]

    obs = []
    for cls in (False, True):
        p = [1.0 - torch.exp(1j * angle(mu, nu)) for mu in range(dims) for nu in range(mu + 1, dims)
             if (nu == t) == cls]
        m = sum(x.mean() for x in p) / len(p) if p else torch.zeros((), dtype=torch.complex128)
        obs += [float(m.real), float(m.imag)]
    poly = torch.exp(1j * th[t].sum(dim=0)).mean()
    obs += [float(poly.real), float(poly.imag)]
    if case["multihit"]:
        S = torch.zeros_like(th[0], dtype=torch.complex128)
        U = torch.exp(1j * th)
        for nu in range(t):
            up = _at(U[nu], t) * _at(U[t], nu).conj() * U[nu].conj()
            lo = _at(_at(U[nu], t), nu, -1).conj() * _at(U[t], nu, -1).conj() * _at(U[nu], nu, -1)
            S = S + case["aniso"] * (up + lo)
        a = S.abs()
        x = case["beta"] * a
        field = torch.prod(S.conj() / a * torch.special.i1e(x) / torch.special.i0e(x), dim=0)
    else:
        field = torch.exp(1j * th[t].sum(dim=0))
    R = ext[0] // 2
    corr = [sum((field * _at(field, i, r).conj()).mean() for i in range(t)) / t for r in range(1, R + 1)]
    return {"observables": np.array(obs), "correlator": torch.stack(corr).cpu().numpy()}


def _exact_action(case, seed):
    dims = case["dims"]
    n = dims * _volume(_N(case))
    flat = _angles(case["batch"] * n, seed, getattr(torch, case["dtype"])).reshape(case["batch"], n).double()
    flat.requires_grad_()
    th, _ = _natural(flat, dims, _N(case))
    S = 0.0
    for mu in range(dims):
        for nu in range(mu + 1, dims):
            a, b = th[:, mu], th[:, nu]
            w = case["aniso"] if nu == dims - 1 else 1.0 / case["aniso"]
            S = S + w * (1.0 - torch.cos(a + _at(b, mu) - _at(a, nu) - b)).flatten(1).sum(1)
    S = case["beta"] * S
    (force,) = torch.autograd.grad(S.sum(), flat)
    return {"action": S.detach(), "force": force}


def _exact_layer(th, mu, off, K, w, inverse=False):
    """A coupling layer in 64 bits (w: its four weights, already rounded to bfloat16)."""
    B, _, L, _ = th.shape
    P = th[:, 0] + torch.roll(th[:, 1], -1, -1) - torch.roll(th[:, 0], -1, -2) - th[:, 1]
    r = torch.arange(L, device=th.device)
    frozen = ((r - off) % 4 == 1) | ((r - off) % 4 == 2)
    frozen = frozen[:, None].expand(L, L) if mu == 0 else frozen[None, :].expand(L, L)
    ctx = torch.stack([torch.cos(P), torch.sin(P)], 1) * frozen
    h = F.leaky_relu(F.conv2d(F.pad(ctx, (1, 1, 1, 1), mode="circular"), w[0], w[1]))
    at = torch.nonzero((r - off) % 4 == 0).flatten() if mu == 0 else torch.nonzero((r - off + 1) % 4 == 0).flatten()
    prm = F.conv2d(F.pad(h, (1, 1, 1, 1), mode="circular"), w[2], w[3])
    prm, Pa = (prm[:, :, at], P[:, at]) if mu == 0 else (prm[:, :, :, at], P[:, :, at])
    alpha, wt, shift = torch.exp(prm[:, :K].clamp(-8, 8)), torch.softmax(prm[:, K:2 * K], 1), prm[:, 2 * K]
    two_pi = 2 * math.pi

    def wrap(x):
        return x - two_pi * torch.round(x.detach() / two_pi)

    def mixture(x):
        sn, cs = torch.sin(x / 2)[:, None], torch.cos(x / 2)[:, None]
        g = 2 * torch.atan2(alpha * sn, cs)
        return (wt * g).sum(1), (wt * alpha / (cs * cs + alpha * alpha * sn * sn)).sum(1)

    if inverse:
        z = wrap(Pa - shift)
        with torch.no_grad():
            lo, hi = torch.full_like(z, -math.pi), torch.full_like(z, math.pi)
            for _ in range(60):
                mid = (lo + hi) / 2
                below = mixture(mid)[0] < z
                lo, hi = torch.where(below, mid, lo), torch.where(below, hi, mid)
            x = (lo + hi) / 2
        H, Hp = mixture(x)
        x = x - (H - z) / Hp.detach()  # the solution, with its first derivatives
        delta, logd = x - z - shift, torch.log(mixture(x)[1])
    else:
        xc = wrap(Pa)
        H, Hp = mixture(xc)
        delta, logd = H + shift - xc, torch.log(Hp)
    full = torch.zeros_like(th[:, 0])
    if mu == 0:
        full = full.index_copy(1, at, delta)
        out = torch.stack([th[:, 0] + full, th[:, 1]], 1)
    else:
        full = full.index_copy(2, (at + 1) % L, delta)
        out = torch.stack([th[:, 0], th[:, 1] + full], 1)
    return out, logd.flatten(1).sum(1)


def _exact_weights(K, hidden, seed):
    net = torch.nn.Sequential(torch.nn.Conv2d(2, hidden, 3), torch.nn.LeakyReLU(),
                              torch.nn.Conv2d(hidden, 2 * K + 1, 3)).to(DEVICE)
    _weights(net, seed)
    return [p.detach().bfloat16().double().requires_grad_() for p in net.parameters()]


def _exact_flow_layer(case, seed):
    x = _flow_inputs(case, seed)
    w = _exact_weights(case["K"], case["hidden"], seed)
    outs, grads = [[], []], None
    for k in range(0, case["batch"], 128):  # a slice of the batch at a time: weight gradients add up
        th = x["theta"][k:k + 128].double().requires_grad_()
        out, ld = _exact_layer(th, case["mu"], case["off"], case["K"], w, case["inverse"])
        g = torch.autograd.grad([out, ld], [th] + w,
                                [x["g_theta"][k:k + 128].double(), x["g_logdet"][k:k + 128].double()])
        grads = [[g[0]]] + list(g[1:]) if grads is None else \
            [grads[0] + [g[0]]] + [a + b for a, b in zip(grads[1:], g[1:])]
        outs[0].append(out.detach())
        outs[1].append(ld.detach())
    return {"theta": torch.cat(outs[0]), "logdet": torch.cat(outs[1]), "grads": [torch.cat(grads[0])] + grads[1:]}


@torch.no_grad()
def _exact_flow_sample(case, seed):
    L = case["L"]
    th = (torch.rand((case["batch"], 2, L, L), device=DEVICE, generator=_generator(seed)) * (2 * math.pi)).double()
    logq = torch.full((case["batch"],), -2 * L * L * math.log(2 * math.pi), dtype=torch.float64, device=DEVICE)
    for k in range(case["layers"]):
        w = _exact_weights(case["K"], case["hidden"], 100 * int(seed) + k)
        th, ld = _exact_layer(th, k % 2, (k // 2) % 4, case["K"], w)
        logq = logq - ld
    return {"cos": torch.cos(th), "sin": torch.sin(th), "logq": logq}
