"""Which route a sweep takes, by the kernels it launches: links are the same on
every route, so only the count tells whether the cluster or the two-phase
kernels ran or a fallback did.

One launch per phase: 2 dims (metrop + ovrn).  Cluster: one for the sweep.  Two
phases per launch: per half-pass 2 of 4 launches (4D) where both pairs of
directions fit a block, 3 where one does, 2 of 3 in 3D."""
from __future__ import annotations

import pytest

pytestmark = pytest.mark.gpu


def _launches(lat, rng, metrop=1, ovrn=2):
    from latticeu1_b200 import launch_count
    n = launch_count()
    lat.update(rng, metrop, ovrn)
    return launch_count() - n


# the smallest lattices, one block and sixteen, the largest of the route, and the
# first ones beyond it (None): 1024 sites a block in 2D and 3D, 704 in 4D
@pytest.mark.parametrize("dims,N,cluster", [
    (2, (4, 0, 0, 4), True), (2, (32, 0, 0, 32), True), (2, (34, 0, 0, 32), True), (2, (128, 0, 0, 256), True),
    (2, (130, 0, 0, 256), False), (3, (2, 2, 0, 2), True), (3, (32, 32, 0, 32), True), (3, (32, 34, 0, 32), False),
    (4, (2, 2, 2, 2), True), (4, (8, 8, 8, 8), True), (4, (10, 12, 14, 12), True), (4, (22, 8, 8, 16), True),
    (4, (12, 12, 12, 14), False)])
@pytest.mark.parametrize("window", [None, (0.7, 3)])
def test_cluster_route_is_taken(ctx, dims, N, cluster, window, monkeypatch):
    from latticeu1_b200 import Lattice, Rng
    monkeypatch.setenv("U1_TUNE", "0")
    monkeypatch.delenv("U1_CLUSTER", raising=False)
    lat, rng = Lattice(ctx, dims, N, 1.1), Rng(ctx, 5)
    if window:
        lat.set_metropolis(*window)
    lat.hot_start(rng)
    for _ in range(2):
        assert _launches(lat, rng) == (1 if cluster else 2 * dims * 3)
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


@pytest.mark.parametrize("dims,N,tuned", [(4, (8, 8, 8, 8), False), (2, (32, 0, 0, 32), False),
                                          (4, (16, 16, 16, 16), True)])
def test_only_phase_kernels_are_tuned(ctx, dims, N, tuned, monkeypatch, tmp_path):
    """The first update of a lattice on the cluster route times nothing: no trial, no line in the cache."""
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
    lat.close()
