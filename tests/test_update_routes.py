"""Routes a sweep can take: the four-site kernel at rows that do and do not
divide a warp, and the one-launch cluster sweep of small lattices, against the
one-site kernel.  All routes do the same arithmetic in the same order, so the
links are compared bit for bit."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    from latticeu1_b200 import Context
    return Context(0)


def _chain(ctx, dims, N, aniso, variant, block=0, window=None, sweeps=((1, 2), (2, 0), (0, 1))):
    import torch

    from latticeu1_b200 import Lattice, Rng
    lat = Lattice(ctx, dims, N, 1.1, aniso)
    if variant:
        lat.set_variant(variant)
    if block:
        lat.set_block(block)
    if window:
        lat.set_metropolis(*window)
    rng = Rng(ctx, 31)
    lat.hot_start(rng)
    for m, o in sweeps:
        lat.update(rng, m, o)
    obs = torch.zeros(6, dtype=torch.float64, device="cuda")
    lat.update_measure(rng, 1, 1, obs.data_ptr())
    torch.cuda.synchronize()
    out = lat.export_angles(), obs.cpu().numpy().copy(), rng.state
    ref = lat.measure()
    lat.close()
    flat = np.array([f(ref[k]) for k in ("plaq_ss", "plaq_st", "poly") for f in (np.real, np.imag)])
    # the measurement of the same links, summed in FP64 from FP32 terms of a few sites
    assert np.nanmax(np.abs(out[1] - flat)) < 1e-6  # 2D has no spatial plaquettes: NaN
    return out


# x0-rows of 1, 2, 3, 5, 6, 8, 12 and 33 quads: within a warp, across warps,
# longer than a warp; the last block partly filled
@pytest.mark.parametrize("dims,N", [
    (4, (8, 6, 4, 6)), (4, (16, 4, 6, 4)), (4, (24, 4, 4, 6)), (4, (40, 6, 4, 4)), (4, (48, 4, 6, 4)),
    (3, (64, 6, 0, 10)), (3, (96, 4, 0, 6)), (2, (264, 0, 0, 6))])
@pytest.mark.parametrize("block", [64, 128])
def test_four_site_rows(ctx, dims, N, block):
    a = _chain(ctx, dims, N, 1.5, 5, block)
    b = _chain(ctx, dims, N, 1.5, 3)
    assert np.array_equal(a[0], b[0]) and a[2] == b[2]


# one block (up to 512 sites of a parity) and sixteen, shares that do not divide
# the rows (idle and short blocks), the smallest extents, the largest lattices
# of the route and the first ones beyond it
@pytest.mark.parametrize("dims,N", [
    (2, (4, 0, 0, 4)), (2, (32, 0, 0, 32)), (2, (34, 0, 0, 32)), (2, (62, 0, 0, 46)), (2, (128, 0, 0, 256)),
    (2, (130, 0, 0, 256)), (2, (2048, 0, 0, 16)), (3, (2, 2, 0, 2)), (3, (10, 6, 0, 14)), (3, (32, 32, 0, 32)),
    (4, (2, 2, 2, 2)), (4, (8, 8, 8, 2)), (4, (6, 10, 8, 4)), (4, (8, 8, 8, 8)), (4, (10, 12, 14, 12)),
    (4, (22, 8, 8, 16)), (4, (22, 8, 16, 8))])
@pytest.mark.parametrize("window", [None, (0.7, 3)])
def test_cluster_sweep(ctx, dims, N, window, monkeypatch):
    monkeypatch.setenv("U1_TUNE", "0")
    a = _chain(ctx, dims, N, 0.8, 0, window=window)
    b = _chain(ctx, dims, N, 0.8, 3, window=window)
    assert np.array_equal(a[0], b[0]) and a[2] == b[2]


def test_cluster_sweep_in_multilevel(ctx, monkeypatch):
    """Frozen time slices, the work copy of the links, graphs on and off."""
    from latticeu1_b200 import Lattice, Rng
    monkeypatch.setenv("U1_TUNE", "0")
    res = []
    for variant, graphs in ((0, True), (0, False), (3, True)):
        lat = Lattice(ctx, 4, (6, 4, 8, 12), 0.95)
        if variant:
            lat.set_variant(variant)
        lat.set_graphs(graphs)
        rng = Rng(ctx, 3)
        lat.hot_start(rng)
        res.append((lat.multilevel(rng, 2, 1, 3, 2, 1, 2), lat.export_angles(), rng.state))
        lat.close()
    for r in res[1:]:
        assert np.array_equal(r[0], res[0][0]) and np.array_equal(r[1], res[0][1]) and r[2] == res[0][2]


# planes and diagonals of one to several blocks, partly filled blocks, the largest
# plane (512 sites), diagonals that are too long (22 x 18 x 14 x 30: only the planes
# pair up), Nx/2 odd, extents of 2
DUO = [(4, (8, 4, 6, 6)), (4, (4, 8, 2, 2)), (4, (16, 16, 16, 16)), (4, (6, 10, 12, 4)), (4, (22, 18, 14, 30)),
       (4, (64, 16, 4, 6)), (4, (20, 20, 20, 20)), (4, (10, 12, 32, 16)), (3, (40, 18, 0, 22)), (3, (2, 4, 0, 6)),
       (3, (34, 30, 0, 10))]


# four sites per thread: rows of one to sixteen quads, rows that cross warps (24, 40),
# extents of 2, partly filled blocks, blocks of 288 (the last), planes of up to 1024 threads; register bounds 96
# (few blocks), 72 (64 x 64 x 4 x 2; several waves of 288 threads) and 64 (planes above
# 896 threads; several waves of 512, links above half the L2)
QUAD_DUO = [(4, (8, 2, 2, 2)), (4, (8, 4, 4, 6)), (4, (16, 16, 16, 16)), (4, (24, 24, 4, 6)), (4, (40, 40, 4, 4)),
            (4, (64, 64, 4, 2)), (4, (128, 64, 4, 4)), (4, (8, 4, 34, 34)), (4, (48, 48, 24, 20)),
            (4, (64, 64, 24, 24)), (3, (16, 10, 0, 6)), (3, (32, 34, 0, 38)), (4, (16, 24, 6, 4)), (4, (24, 16, 6, 4)),
            (4, (24, 24, 6, 10))]


def _duo_child(out, geometries=None):
    """Every geometry with two phases per launch (as cached by the tuner) and with the one-site kernel."""
    from latticeu1_b200 import Context, Lattice, Rng
    ctx = Context(0)
    res = {}
    for k, (dims, N) in enumerate(geometries or DUO):
        for window in (None, (0.7, 3)):
            a = _chain(ctx, dims, N, 0.8, 0, window=window)
            b = _chain(ctx, dims, N, 0.8, 3, window=window)
            res[f"{k}_{window is None}"] = np.array([np.array_equal(a[0], b[0]), a[2] == b[2]])
    ml = []
    for variant in (0, 3):
        lat = Lattice(ctx, 4, (16, 16, 16, 16), 0.95)
        if variant:
            lat.set_variant(variant)
        rng = Rng(ctx, 3)
        lat.hot_start(rng)
        lat.update(rng, 1, 1)
        ml.append((lat.multilevel(rng, 1, 1, 2, 1, 1, 2), lat.export_angles()))
    res["multilevel"] = np.array([np.array_equal(ml[0][0], ml[1][0]), np.array_equal(ml[0][1], ml[1][1])])
    np.savez(out, **res)


@pytest.mark.parametrize("variant,geometries", [(3, "DUO"), (5, "QUAD_DUO")])
def test_two_phases_per_launch(ctx, tmp_path, variant, geometries):
    import os
    import subprocess
    import sys
    from pathlib import Path

    import torch
    name = torch.cuda.get_device_name(0)
    lines = []
    for k, (dims, N) in enumerate(globals()[geometries]):
        g = {3: (N[0], N[1], N[3], 1), 4: N}[dims]
        lines.append(f"{name}|update|{dims}|{'x'.join(map(str, g))}\t{variant}\t1.0\t{(128, 192, 256)[k % 3]}\t1\n")
    (tmp_path / "u1b200_tunecache.tsv").write_text("".join(lines))
    root = Path(__file__).resolve().parent.parent
    env = dict(os.environ, U1_RESOURCE_PATH=str(tmp_path), U1_CLUSTER="0", PYTHONPATH=f"{root}:{root / 'tests'}")
    env.pop("U1_TUNE", None)
    out = tmp_path / "r.npz"
    code = f"import test_update_routes as t; t._duo_child({str(out)!r}, t.{geometries})"
    subprocess.run([sys.executable, "-c", code], env=env, check=True, timeout=300)
    assert (tmp_path / "u1b200_tunecache.tsv").read_text() == "".join(lines)  # every geometry came from the cache
    for k, v in np.load(out).items():
        assert v.all(), (k, v)
