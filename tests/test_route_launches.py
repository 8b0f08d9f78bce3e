"""Which route a sweep takes, by the kernels it launches: links are the same on
every route, so only the count tells whether the cluster or the two-phase
kernels ran or a fallback did.

One launch per phase: 2 dims (metrop + ovrn).  Cluster: one for the sweep.  Two
phases per launch: per half-pass 2 of 4 launches (4D) where both pairs of
directions fit a block, 3 where one does, 2 of 3 in 3D."""
from __future__ import annotations

import os
import subprocess
import sys
from pathlib import Path

import numpy as np
import pytest

ROOT = Path(__file__).resolve().parents[1]
for p in (ROOT, ROOT / "tests"):
    if str(p) not in sys.path:
        sys.path.insert(0, str(p))

pytestmark = pytest.mark.gpu


def _launches(lat, rng, metrop=1, ovrn=2):
    from latticeu1_b200 import launch_count
    n = launch_count()
    lat.update(rng, metrop, ovrn)
    return launch_count() - n


# the smallest lattices, one block and sixteen, the largest of the route: 1024
# sites a block in 2D and 3D, 704 in 4D
CLUSTER = [(2, (4, 0, 0, 4), 1), (2, (32, 0, 0, 32), 1), (2, (34, 0, 0, 32), 1), (2, (62, 0, 0, 46), 1),
           (2, (128, 0, 0, 256), 1), (3, (2, 2, 0, 2), 1), (3, (10, 6, 0, 14), 1), (3, (32, 32, 0, 32), 1),
           (4, (2, 2, 2, 2), 1), (4, (8, 8, 8, 8), 1), (4, (6, 10, 8, 4), 1), (4, (10, 12, 14, 12), 1),
           (4, (22, 8, 8, 16), 1)]
# and the first ones beyond it
BEYOND = [(2, (130, 0, 0, 256), 12), (3, (32, 34, 0, 32), 18), (4, (12, 12, 12, 14), 24)]

# the geometries of test_update_routes with the launches of a half-pass, one and
# four sites per thread: directions 2, 3 pair up in no four-site launch, and with
# one site where diagonals of lcm(N2, N3) sites, eight or more side by side, fit 256 threads
DUO_LAUNCHES = [2, 2, 2, 2, 3, 2, 2, 3, 2, 2, 2]
QUAD_DUO_LAUNCHES = [3] * 10 + [2, 2] + [3] * 3


def half_pass_launches(route):
    import test_update_routes as t
    geometries, counts = (t.DUO, DUO_LAUNCHES) if route == "duo" else (t.QUAD_DUO, QUAD_DUO_LAUNCHES)
    assert len(geometries) == len(counts)
    return [(dims, N, n) for (dims, N), n in zip(geometries, counts)]


def cache_lines(route):
    """A tune-cache file that names two phases per launch for every geometry of the route."""
    import torch
    name, variant, lines = torch.cuda.get_device_name(0), 3 if route == "duo" else 5, []
    for k, (dims, N, _) in enumerate(half_pass_launches(route)):
        g = {3: (N[0], N[1], N[3], 1), 4: N}[dims]
        lines.append(f"{name}|update|{dims}|{'x'.join(map(str, g))}\t{variant}\t1.0\t{(128, 192, 256)[k % 3]}\t1\n")
    return "".join(lines)


@pytest.mark.parametrize("dims,N,launches", CLUSTER + BEYOND)
@pytest.mark.parametrize("window", [None, (0.7, 3)])
def test_cluster_route_is_taken(ctx, dims, N, launches, window, monkeypatch):
    from latticeu1_b200 import Lattice, Rng
    monkeypatch.setenv("U1_TUNE", "0")
    monkeypatch.delenv("U1_CLUSTER", raising=False)
    lat, rng = Lattice(ctx, dims, N, 1.1), Rng(ctx, 5)
    if window:
        lat.set_metropolis(*window)
    lat.hot_start(rng)
    for _ in range(2):
        assert _launches(lat, rng) == launches
    lat.close()


def test_block_size_selects_the_phase_kernels(ctx, monkeypatch):
    """An explicit block size is a request for the kernels it applies to, as an explicit variant is."""
    from latticeu1_b200 import Lattice, Rng
    monkeypatch.setenv("U1_TUNE", "0")
    monkeypatch.delenv("U1_CLUSTER", raising=False)
    lat, rng = Lattice(ctx, 4, (8, 8, 8, 8), 1.1), Rng(ctx, 5)
    lat.hot_start(rng)
    assert _launches(lat, rng) == 1
    lat.set_block(64)
    assert _launches(lat, rng) == 24 and lat.block == 64
    lat.set_variant(0)
    assert _launches(lat, rng) == 1
    lat.set_variant(3)
    assert _launches(lat, rng) == 24
    lat.tune(rng)  # gives the choice back
    assert _launches(lat, rng) == 1
    lat.close()


# both sides of the lines between the cluster and the tuned phase kernels: one block,
# 3D at 768 sites a block, 4D at 192 (two pairs of directions), 512 (one) and 704 (none)
@pytest.mark.parametrize("dims,N,tuned", [
    (4, (8, 8, 8, 8), False), (2, (32, 0, 0, 32), False), (2, (128, 0, 0, 256), False), (4, (6, 6, 6, 4), False),
    (3, (28, 28, 0, 30), False), (3, (26, 30, 0, 32), True), (3, (32, 32, 0, 32), True),
    (4, (8, 8, 8, 12), False), (4, (8, 8, 10, 10), True), (4, (12, 12, 12, 12), True),
    (4, (12, 8, 14, 12), False), (4, (10, 10, 12, 14), True), (4, (64, 36, 2, 2), False),
    (4, (16, 16, 16, 16), True)])
def test_only_phase_kernels_are_tuned(ctx, dims, N, tuned, monkeypatch, tmp_path):
    """The cluster route up to where the tuned phase kernels overtake it; there the first update times
    nothing: no trial, no line in the cache."""
    from latticeu1_b200 import Lattice, Rng
    monkeypatch.setenv("U1_RESOURCE_PATH", str(tmp_path))
    monkeypatch.delenv("U1_TUNE", raising=False)
    monkeypatch.delenv("U1_CLUSTER", raising=False)
    lat, rng = Lattice(ctx, dims, N, 1.1), Rng(ctx, 5)
    lat.hot_start(rng)
    n = _launches(lat, rng)
    lines = [p.read_text() for p in tmp_path.glob("u1b200_tunecache.tsv")]
    if tuned:
        # another test of this process may have tuned the geometry already: then it is taken from memory
        assert n > 1 and len(lines) <= 1
    else:
        assert n == 1 and not lines
    assert lat.variant in (1, 2, 3, 5)
    ref, rng_ref = Lattice(ctx, dims, N, 1.1), Rng(ctx, 5)
    ref.set_variant(3)
    ref.hot_start(rng_ref)
    _launches(ref, rng_ref)
    assert np.array_equal(lat.export_angles(), ref.export_angles())
    lat.close()
    ref.close()


def test_multilevel_of_an_untuned_lattice(ctx, monkeypatch):
    """Sub-updates before and after a lattice beyond the line is tuned: another route, the same numbers."""
    from latticeu1_b200 import Lattice, Rng
    monkeypatch.delenv("U1_TUNE", raising=False)
    monkeypatch.delenv("U1_CLUSTER", raising=False)
    out = []
    for variant, update in ((0, False), (0, True), (3, False)):
        lat, rng = Lattice(ctx, 4, (8, 8, 10, 12), 0.95), Rng(ctx, 3)
        if variant:
            lat.set_variant(variant)
        lat.hot_start(rng)
        first = lat.multilevel(rng, 1, 1, 2, 1, 1, 1)
        if update:
            lat.tune(rng)
        out.append((first, lat.multilevel(rng, 1, 1, 2, 1, 1, 1), lat.export_angles(), rng.state))
        lat.close()
    for o in out[1:]:
        assert np.array_equal(o[0], out[0][0]) and np.array_equal(o[1], out[0][1])
        assert np.array_equal(o[2], out[0][2]) and o[3] == out[0][3]


def test_tuned_lattice_continues_its_chain(ctx, monkeypatch, tmp_path):
    """A lattice beyond the cluster route after tune(): the tuned kernels run, and give the untuned one's links."""
    from latticeu1_b200 import Lattice, Rng
    monkeypatch.setenv("U1_RESOURCE_PATH", str(tmp_path))
    monkeypatch.delenv("U1_CLUSTER", raising=False)
    a, b = (Lattice(ctx, 4, (16, 16, 16, 8), 1.0) for _ in range(2))
    ra, rb = Rng(ctx, 5), Rng(ctx, 5)
    for lat, rng in ((a, ra), (b, rb)):
        lat.set_variant(3)
        lat.hot_start(rng)
        lat.update(rng, 1, 2)
    a.tune(ra)
    assert 12 <= _launches(a, ra) <= 24 and _launches(b, rb) == 24
    assert np.array_equal(a.export_angles(), b.export_angles()) and ra.state == rb.state
    # another lattice of the geometry, left automatic, takes the choice over
    c, rc = Lattice(ctx, 4, (16, 16, 16, 8), 1.0), Rng(ctx, 6)
    c.hot_start(rc)
    assert _launches(c, rc) == _launches(a, ra) and (c.variant, c.block) == (a.variant, a.block)


def test_bench_chains_share_the_tuned_route(ctx, monkeypatch):
    """The end-to-end chains beside the first one are left to the automatic choice: a variant and a block
    size set from the first would run one phase per launch where it runs two."""
    from types import SimpleNamespace

    import torch

    import bench
    from latticeu1_b200 import Lattice, Rng
    N = (16, 16, 16, 16)
    lat, rng, stream = Lattice(ctx, 4, N, 1.0), Rng(ctx, 5), torch.cuda.Stream()
    lat.set_stream(stream.cuda_stream)
    lat.hot_start(rng)
    lat.update(rng, 1, 4)
    lat.synchronize()

    def refuse(*a):
        raise AssertionError("an automatic chain was given an explicit kernel")

    monkeypatch.setattr(Lattice, "set_variant", refuse)
    monkeypatch.setattr(Lattice, "set_block", refuse)
    args = SimpleNamespace(delta=0.0, nhits=1, variant=0, block=0, steps=2)
    rate, steps, finite = bench.e2e_rate(ctx, lat, rng, stream, N, 1.0, 1.0, args, 0, 1)
    assert rate > 0 and steps == 6 and finite


def _child(route):
    from latticeu1_b200 import Context, Lattice, Rng
    ctx = Context(0)
    for dims, N, per in half_pass_launches(route):
        lat, rng = Lattice(ctx, dims, N, 0.8), Rng(ctx, 3)
        lat.hot_start(rng)
        for _ in range(2):
            n = _launches(lat, rng)
            assert n == per * 2 * 3, (dims, N, n, per)
        lat.close()
    print("LAUNCHES_OK")


@pytest.mark.parametrize("route", ["duo", "quad"])
def test_two_phases_per_launch_are_launched(route, tmp_path):
    (tmp_path / "u1b200_tunecache.tsv").write_text(cache_lines(route))
    env = dict(os.environ, PYTHONPATH=f"{ROOT}:{ROOT / 'tests'}", U1_RESOURCE_PATH=str(tmp_path), U1_CLUSTER="0")
    env.pop("U1_TUNE", None)
    r = subprocess.run([sys.executable, "-c", f"import test_route_launches as t; t._child({route!r})"], env=env,
                       capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and "LAUNCHES_OK" in r.stdout, (r.stdout[-3000:], r.stderr[-3000:])
