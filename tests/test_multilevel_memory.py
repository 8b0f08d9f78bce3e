"""Multilevel on a device whose memory holds the tensors of one sub-update but
not a batch of slab products beside them: the call falls back to one sub-update
a batch and gives the same numbers.  The shortage is made on the host, by an
allocator (u1_set_device_allocator) with a budget; a child process, so that no
other test's objects hold memory from it."""
from __future__ import annotations

import os
import subprocess
import sys
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parents[1]
N = (16, 16, 16, 16)


def _child() -> None:
    import numpy as np
    import torch

    from latticeu1_b200 import Context, Lattice, Rng, U1Error, _lib
    torch.cuda.init()
    live, st = {}, {"budget": None, "refused": 0}

    def alloc(user, nbytes, out):
        if st["budget"] is not None and sum(live.values()) + nbytes > st["budget"]:
            st["refused"] += 1
            return 1
        p = torch.cuda.caching_allocator_alloc(max(int(nbytes), 1), device=0)
        live[p] = nbytes
        out[0] = p
        return 0

    def release(user, p):
        live.pop(p)
        torch.cuda.caching_allocator_delete(p)

    a_fn, r_fn = _lib.DEV_ALLOC_FN(alloc), _lib.DEV_FREE_FN(release)
    _lib.check(_lib.lib.u1_set_device_allocator(a_fn, r_fn, None), "u1_set_device_allocator")
    ctx = Context(0)
    Vs, R, nl2, nl4 = N[0] * N[1] * N[2], N[0] // 2, N[3] // 2, N[3] // 4
    slab, t2, t4 = 16 * Vs * nl2, 16 * Vs * R * 3 * nl2, 16 * Vs * R * 3 * nl4
    work, small = 32 * Vs * N[3], 1 << 20  # small: partial sums
    results = []
    one, batch = work + slab + t2 + t4, work + 16 * slab + t2 + t4
    # no limit; T2 refused beside the batch; T4 refused; one byte less than one sub-update needs
    for budget in (None, one + small, batch - 1, one - 1):
        lat, rng = Lattice(ctx, 4, N, 0.95), Rng(ctx, 3)
        lat.hot_start(rng)
        lat.update(rng, 1, 1)
        held = sum(live.values())
        st["budget"] = None if budget is None else held + budget
        st["refused"] = 0
        try:
            corr = lat.multilevel(rng, 2, 1, 19, 1, 1, 1)
            assert st["refused"] == (0 if budget is None else 1), (budget, st)
        except U1Error as e:
            assert budget == one - 1 and e.code == _lib.U1_ERR_NOMEM, (budget, e)
            assert sum(live.values()) == held  # nothing kept
            corr = None
        st["budget"] = None
        if corr is not None:
            results.append((corr, lat.export_angles()))
        lat.close()
        rng.close()
        torch.cuda.synchronize()
        assert not live and _lib.device_allocations() == 0, budget
    for r in results[1:]:
        assert np.array_equal(r[0], results[0][0]) and np.array_equal(r[1], results[0][1])
    assert len(results) == 3
    _lib.check(_lib.lib.u1_set_device_allocator(_lib.NO_ALLOC, _lib.NO_FREE, None), "u1_set_device_allocator")
    print("MEMORY_OK")


@pytest.mark.gpu
def test_short_of_memory_for_a_batch():
    env = {**os.environ, "PYTHONPATH": str(ROOT), "U1_TUNE": "0"}
    r = subprocess.run([sys.executable, str(Path(__file__).resolve()), "child"], cwd=str(ROOT), env=env,
                       capture_output=True, text=True, timeout=600)
    assert r.returncode == 0 and "MEMORY_OK" in r.stdout, (r.stdout[-3000:], r.stderr[-3000:])


if __name__ == "__main__" and sys.argv[1:] == ["child"]:
    sys.path.insert(0, str(ROOT))
    try:
        _child()
    except BaseException:
        import traceback
        traceback.print_exc()
        sys.stderr.flush()
        os._exit(1)  # objects that still hold memory of the Python allocator must not be torn down after it
