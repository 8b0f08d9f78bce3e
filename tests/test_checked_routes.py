"""The two-phase kernels and the cluster sweep in the checked build
(U1_CHECKED=1): every link access in bounds and aligned, no link read or written
by two blocks that a launch stores, every shared-memory address of the cluster
sweep inside its row, and the links those of the one-site kernel.  A child
process per route takes the two-phase layouts from a tune-cache file, as a
user's lattice takes the tuner's choice."""
from __future__ import annotations

import json
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

from test_route_launches import CLUSTER, cache_lines, half_pass_launches  # noqa: E402


def _child(route: str) -> None:
    from latticeu1_b200 import Context, Lattice, Rng, _lib, launch_count
    assert _lib.CHECKED
    ctx = Context(0)
    out = {"selftest": _lib.check_selftest(ctx.handle), "cases": []}
    for dims, N, per in CLUSTER if route == "cluster" else half_pass_launches(route):
        for window in (None, (0.7, 3)):
            links, phases, got = [], 0, 0
            for variant in (0, 3):
                lat, rng = Lattice(ctx, dims, N, 0.8, 1.2), Rng(ctx, 31)
                if variant:
                    lat.set_variant(variant)
                if window:
                    lat.set_metropolis(*window)
                lat.hot_start(rng)
                n = launch_count()
                for m, o in ((1, 2), (2, 0)):
                    lat.update(rng, m, o)
                if variant == 0:
                    got = launch_count() - n
                    phases = 0 if route == "cluster" else per * 2 * 5
                    out["cases"].append([dims, N, _lib.check_report(ctx.handle, reset=True), got, phases])
                links.append(lat.export_angles())
                lat.close()
                rng.close()
            out["cases"][-1].append(bool(np.array_equal(*links)))
            _lib.check_report(ctx.handle, reset=True)
    print(json.dumps(out))


@pytest.mark.gpu
@pytest.mark.parametrize("route", ["cluster", "duo", "quad"])
def test_checked_route(route, tmp_path):
    env = dict(os.environ, PYTHONPATH=f"{ROOT}:{ROOT / 'tests'}", U1_CHECKED="1", U1_RESOURCE_PATH=str(tmp_path),
               U1_CLUSTER="1" if route == "cluster" else "0")
    env.pop("U1_TUNE", None)
    if route == "cluster":
        env["U1_TUNE"] = "0"  # the route to its largest lattices
    else:
        (tmp_path / "u1b200_tunecache.tsv").write_text(cache_lines(route))
    r = subprocess.run([sys.executable, str(Path(__file__).resolve()), route], cwd=str(ROOT), env=env,
                       capture_output=True, text=True, timeout=900)
    assert r.returncode == 0, (r.stdout[-3000:], r.stderr[-3000:])
    out = json.loads([ln for ln in r.stdout.splitlines() if ln.startswith("{")][-1])
    assert out["cases"]
    for dims, N, rep, launches, phases, same in out["cases"]:
        where = (dims, N, rep)
        assert rep["bad"] == 0 and rep["races"] == 0, where
        assert same, where
        if route == "cluster":
            assert launches == 2 and rep["phases"] == 0, (where, launches)
        else:
            # a checked launch each; with no overrelaxation pass one more for the rng's pass counter
            assert launches == phases + 1 and rep["phases"] == phases and rep["marked"] > 0, (where, launches, phases)


if __name__ == "__main__" and len(sys.argv) == 2:
    _child(sys.argv[1])
