"""Fused coupling layers of different shapes from several host threads at once:
a kernel's shared-memory limit belongs to the kernel, not to a call, so no call
may lower what another one's launch needs.  The library is called directly, as
often as a thread can; every call must return U1_OK, and the last results are
those that each shape has alone."""
import threading

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("backward", [False, True])
def test_threads_with_different_shapes(backward):
    from latticeu1_b200 import _lib
    K, shapes = 6, [(32, 32, 2), (4, 4, 1), (16, 32, 4), (8, 8, 1)]  # from 100 KB of shared memory to a few
    jobs, keep = [], []
    for k, (L, H, batch) in enumerate(shapes):
        g = torch.Generator("cuda").manual_seed(k)

        def rand(*n, scale=1.0):
            keep.append(torch.randn(*n, device="cuda", generator=g) * scale)
            return keep[-1]

        nw = H * 18 + H + (2 * K + 1) * (H * 9 + 1)
        th, w = rand(batch, 2, L, L, scale=3.0), [rand(n, scale=0.2) for n in (H * 18, H, (2 * K + 1) * H * 9, 2 * K + 1)]
        out, ld, part, wg = rand(batch, 2, L, L), rand(batch), rand(batch, nw), rand(nw)
        stream = torch.cuda.Stream()
        keep.append(stream)
        tail = [batch, L, k % 2, k, K, H, *(t.data_ptr() for t in w), 0.01, stream.cuda_stream]
        if backward:
            g_out = rand(batch, 2, L, L)
            fn, args = _lib.lib.u1_flow_layer_backward, [th.data_ptr(), g_out.data_ptr(), None, out.data_ptr(),
                                                         part.data_ptr(), wg.data_ptr(), *tail]
            results = [out, wg]
        else:
            fn, args = _lib.lib.u1_flow_layer_forward, [th.data_ptr(), out.data_ptr(), ld.data_ptr(), *tail]
            results = [out, ld]
        torch.cuda.synchronize()
        _lib.check(fn(*args), "alone")
        torch.cuda.synchronize()
        jobs.append((fn, args, results, [r.clone() for r in results]))
    codes, start = [], threading.Barrier(len(jobs))

    def work(fn, args):
        start.wait()
        for _ in range(5000):
            rc = fn(*args)
            if rc:
                codes.append((rc, _lib.last_error()))

    threads = [threading.Thread(target=work, args=j[:2]) for j in jobs]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    torch.cuda.synchronize()
    assert not codes, (len(codes), codes[:3])
    for _, _, results, want in jobs:
        assert all(torch.equal(a, b) for a, b in zip(results, want))
