"""Solves that leave a batch part-way (prt_batch_remove) and go on by
themselves (prt_flow_launch, prt_adr_launch): the loop takes up the lattice or
state, the count and the check schedule as the batch left them, so fields,
counts and stop decisions are the single solve's bit for bit, also after an
odd count and off the check interval.  So they are when a finished loop, of its own or a
batch's, is launched once more."""

import contextlib
import ctypes
import io

import numpy as np
import pytest

from golden.fields import integer_velocity

pytestmark = pytest.mark.gpu

# steps of a graph replay: an odd count, one off the check interval, one on it
LEFT = [7, 20, 50]
SMALL, LARGE = 20, 34  # one cluster takes the first
LOOPS = [("0", SMALL, "fp64"), ("1", SMALL, "fp64"), ("1", SMALL, "fp16"), ("1", LARGE, "fp32f")]


def pack(edge, seed=4):
    from prtlb_gpu import random_pack
    return random_pack((edge, edge - 3, edge + 2), 0.5, 2.0, 3.5, seed=seed)


def in_batch(ctx, steps, done=0, remove=True):
    """`steps` steps of the started solve inside a batch, which it then leaves."""
    from prtlb_gpu import _lib
    from prtlb_gpu.batch import Batch
    L = _lib.lib()
    b = Batch(graph_steps=steps, quiet=True)
    try:
        n = ctypes.c_int32()
        b._check(L.prt_batch_add(b.handle, ctx.handle))
        b._check(L.prt_batch_run(b.handle, steps, ctypes.byref(n)))
        assert n.value == done
        if remove:
            b._check(L.prt_batch_remove(b.handle, ctx.handle))
    finally:
        b.close()


def wait(ctx):
    from prtlb_gpu import _lib
    busy = ctypes.c_int32(1)
    while busy.value:
        ctx.check(_lib.lib().prt_ctx_busy(ctx.handle, ctypes.byref(busy)))


def flow(g, precision, nit, tol, left=0, launches=1, remove=True):
    """(field, iterations, converged, change, permeability) of a started solve."""
    from prtlb_gpu import _lib
    from prtlb_gpu.flow import flow_params
    L = _lib.lib()
    g8, p = flow_params(g, g.ndim, "flow", nit, 2e-6, 0.8, 3.0 / 16.0, tol, precision)
    ctx = _lib.Context(0)
    try:
        ctx.check(L.prt_flow_start(ctx.handle, g8.ctypes.data_as(ctypes.c_void_p), ctypes.byref(p)))
        if left:
            in_batch(ctx, left, int(left >= nit), remove)
        for _ in range(launches):
            ctx.check(L.prt_flow_launch(ctx.handle))
            wait(ctx)
        vel, fi = np.empty((3,) + g.shape, np.float32), _lib.FlowInfo()
        ctx.check(L.prt_flow_finish(ctx.handle, vel.ctypes.data_as(ctypes.c_void_p),
                                    ctypes.byref(fi)))
        return vel, fi.iters, fi.converged, fi.change, fi.permeability
    finally:
        ctx.close()


def same_flow(a, b):
    assert a[1:] == b[1:]
    assert np.array_equal(a[0], b[0]), float(np.abs(a[0] - b[0]).max())


@pytest.mark.parametrize("nit,tol", [(333, 0.0), (450, 0.0), (2000, 2e-2)])
@pytest.mark.parametrize("left", LEFT)
@pytest.mark.parametrize("cluster,edge,precision", LOOPS)
def test_flow_goes_on_after_a_batch(monkeypatch, cluster, edge, precision, left, nit, tol):
    g = pack(edge)
    monkeypatch.setenv("PRT_CLUSTER", "0")
    want = flow(g, precision, nit, tol)
    assert want[1] == nit if tol == 0.0 else want[1] < nit
    monkeypatch.setenv("PRT_CLUSTER", cluster)
    same_flow(flow(g, precision, nit, tol, left), want)


def test_flow_of_a_plane_goes_on_after_a_batch():
    g = pack(40)[:, 5]
    same_flow(flow(g, "fp64", 400, 0.0, 7), flow(g, "fp64", 400, 0.0))


@pytest.mark.parametrize("edge", [SMALL, LARGE])
def test_a_finished_flow_loop_launched_again_changes_nothing(edge):
    g = pack(edge)
    same_flow(flow(g, "fp32", 250, 0.0, launches=2), flow(g, "fp32", 250, 0.0))


def test_a_loop_that_a_batch_finished_launched_again_changes_nothing():
    g = pack(SMALL)
    same_flow(flow(g, "fp64", 60, 0.0, 60), flow(g, "fp64", 60, 0.0))


def test_a_flow_that_a_batch_leaves_just_below_its_cap():
    g = pack(LARGE)
    same_flow(flow(g, "fp64", 23, 0.0, 7), flow(g, "fp64", 23, 0.0))


def test_a_flow_goes_on_after_its_batch_was_destroyed():
    g = pack(SMALL)
    same_flow(flow(g, "fp64", 333, 0.0, 20, remove=False), flow(g, "fp64", 333, 0.0))


def transport(g, v, steps, most, left=0, launches=1):
    """(snapshots, times, steps, checks, last remainder) of a started run."""
    from prtlb_gpu import _lib, adr, monod_chemistry
    L = _lib.lib()
    chem = monod_chemistry(0.5)
    ctx = _lib.Context(0)
    try:
        mat8, vel32, geom = adr.stage_inputs(g, v, chem)
        st = _lib.AdrStats()
        ctx.check(L.prt_adr_stage(ctx.handle, mat8.ctypes.data_as(ctypes.c_void_p),
                                  vel32.ctypes.data_as(ctypes.c_void_p), ctypes.byref(geom),
                                  ctypes.byref(st)))
        with contextlib.redirect_stdout(io.StringIO()):
            S = adr.prepare(g.shape, adr.stats_dict(st), 8.0, 1.5, n_species=1, chem=chem, mat=g)
        ctx.check(L.prt_adr_begin(ctx.handle, ctypes.byref(S.params)))
        R = adr.run_params(S, steps, 2e-3, most, 1.12)
        ctx.check(L.prt_adr_start(ctx.handle, ctypes.byref(R)))
        if left:
            assert left % S.check  # it leaves between two checks
            in_batch(ctx, left)
        for _ in range(launches):
            ctx.check(L.prt_adr_launch(ctx.handle))
            wait(ctx)
        r = _lib.AdrResult()
        ctx.check(L.prt_adr_finish(ctx.handle, ctypes.byref(r)))
        ks = adr.ladder_steps(ctx)
        picked = adr.pick(ks, int(r.steps), 4)
        out, t = adr.outputs(ctx, S, 4, int(r.steps), ks, picked, steps, most, {}, 1.5, 0.0)
        return out, t, r.steps, r.checks, r.last_rest
    finally:
        ctx.close()


def same_transport(a, b):
    assert a[2:] == b[2:]
    assert np.array_equal(a[1], b[1])
    assert np.array_equal(a[0], b[0]), float(np.abs(a[0] - b[0]).max())


@pytest.mark.parametrize("steps,most", [(271, 0), (None, 6000)])
@pytest.mark.parametrize("left", [7, 20])
@pytest.mark.parametrize("edge", [SMALL, LARGE])
def test_transport_goes_on_after_a_batch(monkeypatch, edge, left, steps, most):
    g = pack(edge)
    v = integer_velocity(g)
    monkeypatch.setenv("PRT_CLUSTER", "0")
    want = transport(g, v, steps, most)
    assert want[3] > 0
    same_transport(transport(g, v, steps, most, left), want)
    monkeypatch.setenv("PRT_CLUSTER", "1")
    same_transport(transport(g, v, steps, most, left), want)


@pytest.mark.parametrize("edge", [SMALL, LARGE])
def test_a_finished_transport_loop_launched_again_changes_nothing(edge):
    g = pack(edge)
    v = integer_velocity(g)
    same_transport(transport(g, v, 271, 0, launches=2), transport(g, v, 271, 0))
