"""What calls of one process share, what a context gives back, and when the
caller's memory is its own again."""

import ctypes
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_walks_of_two_sizes_side_by_side():
    """Two threads walk grids whose masks need 224 KB and 4 KB of a block's
    shared memory: neither's launch sees the other's size."""
    from prtlb_gpu import _lib, prep
    rng = np.random.default_rng(1)
    grids = [np.where(rng.random(s) < 0.8, 2, 0).astype(np.uint8)
             for s in ((128, 256, 250), (24, 24, 24))]
    want = [prep.inlet_walk(g) for g in grids]
    bad = []

    def many(g, w, n):
        ctx = _lib.Context(0)
        try:
            for _ in range(n):
                got = prep.inlet_walk(g, ctx=ctx)
                if got[1:] != w[1:] or not np.array_equal(got[0], w[0]):
                    bad.append("steps differ")
        except Exception as e:  # pylint: disable=broad-except
            bad.append(repr(e))
        finally:
            ctx.close()

    threads = [threading.Thread(target=many, args=(grids[i % 2], want[i % 2], (12, 300)[i % 2]))
               for i in range(4)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not bad, bad


def test_flow_release_gives_the_memory_back():
    """prt_flow_release frees the lattice, maps and tables whatever their size
    (here under 32 MiB each); a context whose flow phase was ended with
    prt_flow_end solves on with the buffers it kept."""
    from prtlb_gpu import _lib, random_pack
    from prtlb_gpu.flow import flow_params
    from prtlb_gpu.serve import device_memory
    L = _lib.lib()
    g, p = flow_params(random_pack((60, 60, 60), 0.5, 3.0, 5.0, seed=1), 3, "flow", 100, 2e-6, 0.8,
                       3.0 / 16.0, 0.0, "fp32")
    ctx = _lib.Context(0)

    def solve():
        vel = np.empty((3,) + g.shape, np.float32)
        ctx.check(L.prt_flow(ctx.handle, g.ctypes.data_as(ctypes.c_void_p), ctypes.byref(p),
                             vel.ctypes.data_as(ctypes.c_void_p), None))
        return vel

    try:
        solve()
        ctx.check(L.prt_flow_release(ctx.handle))
        before = device_memory(0)[0]
        want = solve()
        assert device_memory(0)[0] <= before - (8 << 20)  # the lattice alone: 8.2 MB
        ctx.check(L.prt_flow_release(ctx.handle))
        assert device_memory(0)[0] == before
        assert np.array_equal(solve(), want)
        ctx.check(L.prt_flow_end(ctx.handle))
        held = before - device_memory(0)[0]
        assert 0 < held <= (40 << 20)  # at most 32 MiB, and the allocator's rounding
        assert np.array_equal(solve(), want)
    finally:
        ctx.close()


def test_a_pinned_result_is_the_callers_again_once_staged():
    """prt_physics_stage has read pinned arrays when it returns: overwriting
    them at once changes nothing of the statistics."""
    import torch
    from prtlb_gpu import _lib
    L = _lib.lib()
    n_t, ns, shape = 6, 4, (128, 128, 96)
    dims = (ctypes.c_int32 * 3)(*shape)
    out = torch.empty((n_t, ns) + shape, dtype=torch.float32, pin_memory=True)
    mat = torch.full(shape, 2, dtype=torch.uint8).pin_memory()
    ctx = _lib.Context(0)
    try:
        for value in (0.25, 0.5, 0.75):
            out.fill_(value)
            ctx.check(L.prt_physics_stage(ctx.handle, ctypes.c_void_p(out.data_ptr()),
                                          ctypes.c_void_p(mat.data_ptr()), 3, dims, n_t, ns))
            out[n_t - 1].fill_(2.0)  # the last to be copied
            st = _lib.PhysicsStats()
            ctx.check(L.prt_physics_stats_dev(ctx.handle, None, None, 3, dims, n_t, ns, 2,
                                              ctypes.byref(st)))
            assert [st.pore_max[j] for j in range(ns)] == [value] * ns
    finally:
        ctx.close()
