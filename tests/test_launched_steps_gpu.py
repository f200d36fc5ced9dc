"""The step launches and their cached loop graphs on grids that one cluster
would take (PRT_CLUSTER=0): every place where a step lets the next one in gives
the same field, a graph follows every change of what it holds, and a batch's
flow steps give the same fields from packed and from plain tables."""

import contextlib
import io

import numpy as np
import pytest

from conftest import load_golden
from test_adr_gpu import adr_kwargs, run

pytestmark = pytest.mark.gpu

RELEASES = [("0", ""), ("1", ""), ("1", "all"), ("1", "none")]
ADR = ["adr_spheres3d_biofilm", "adr_spheres3d_ns4", "adr_spheres3d_monod", "adr_disks2d_first",
       "adr_chan2d_capped"]


@pytest.fixture(autouse=True)
def launches(monkeypatch):
    monkeypatch.setenv("PRT_CLUSTER", "0")


def flow(g, precision, nit=400, tol=1e-9, **kw):
    from prtlb_gpu import stokes_d2q9, stokes_d3q19
    info = {}
    with contextlib.redirect_stdout(io.StringIO()):
        v = (stokes_d3q19 if g.ndim == 3 else stokes_d2q9)(g, nit=nit, tol=tol, info=info,
                                                           precision=precision, **kw)
    return v, info["flow_iters"], info["flow_change"]


def same(a, b):
    assert a[1:] == b[1:] and np.array_equal(a[0], b[0])


@pytest.mark.parametrize("precision", ["fp64", "fp32", "fp32f", "fp16"])
def test_flow_steps_under_every_release(monkeypatch, precision):
    from prtlb_gpu import sphere_pack_3d
    from prtlb_gpu.geometry import disk_pack_2d
    for g in (sphere_pack_3d(24, 0.45, 0), sphere_pack_3d(56, 0.5, 1), disk_pack_2d(40, 0.5, 1)):
        found = []
        for pdl, late in RELEASES:
            monkeypatch.setenv("PRT_PDL", pdl)
            monkeypatch.setenv("PRT_PDL_LATE", late)
            found.append(flow(g, precision))
        for f in found[1:]:
            same(f, found[0])


@pytest.mark.parametrize("pdl,late", RELEASES)
def test_transport_steps_under_every_release(monkeypatch, pdl, late):
    monkeypatch.setenv("PRT_PDL", pdl)
    monkeypatch.setenv("PRT_PDL_LATE", late)
    for name in ADR:
        z = load_golden(name)
        out, tn, info, prog = run(z, name)
        assert np.array_equal(tn, z["t_norm"]), name
        assert np.array_equal(prog, z["progress"]), name
        assert np.array_equal(out, z["out"]), (name, float(np.abs(out - z["out"]).max()))


@pytest.mark.parametrize("pdl,late", RELEASES)
def test_direct_launches_under_every_release(monkeypatch, pdl, late):
    """Without a graph a chunk's first step follows the check kernel in the
    stream; the steps read the control block that it leaves."""
    from prtlb_gpu import sphere_pack_3d
    g = sphere_pack_3d(24, 0.45, 0)
    want = flow(g, "fp64", nit=333, tol=1e-3)
    monkeypatch.setenv("PRT_GRAPHS", "0")
    monkeypatch.setenv("PRT_PDL", pdl)
    monkeypatch.setenv("PRT_PDL_LATE", late)
    same(flow(g, "fp64", nit=333, tol=1e-3), want)
    for name in ADR[2:4]:
        z = load_golden(name)
        out, tn, info, prog = run(z, name)
        assert np.array_equal(prog, z["progress"]), name
        assert np.array_equal(out, z["out"]), (name, float(np.abs(out - z["out"]).max()))


def test_transport_graph_follows_every_change(monkeypatch):
    from prtlb_gpu import _lib, solve_adr
    ctx = _lib.Context(0)

    def solve(name, **change):
        z = load_golden(name)
        with contextlib.redirect_stdout(io.StringIO()):
            return solve_adr(z["mat"], z["vel"], ctx=ctx, **dict(adr_kwargs(z, name), **change))

    try:
        for _ in range(2):
            for name in ADR:
                z = load_golden(name)
                out, tn = solve(name)
                assert np.array_equal(out, z["out"]) and np.array_equal(tn, z["t_norm"]), name
        z = load_golden(ADR[2])
        for pdl in ("0", "1"):
            monkeypatch.setenv("PRT_PDL", pdl)
            assert np.array_equal(solve(ADR[2])[0], z["out"])
        half, _ = solve(ADR[2], steps=adr_kwargs(z, ADR[2])["steps"] // 2)
        full, _ = solve(ADR[2])
        assert np.array_equal(full, z["out"]) and not np.array_equal(half, full)
    finally:
        ctx.close()


def test_flow_graph_follows_every_change(monkeypatch):
    """Solves that differ in grid, porosity at one grid size, precision, force,
    relaxation, count and table alternate on one context; each equals the same
    solve on a context of its own."""
    from prtlb_gpu import _lib, sphere_pack_3d
    from prtlb_gpu.geometry import disk_pack_2d
    a, b, c = sphere_pack_3d(24, 0.45, 0), sphere_pack_3d(24, 0.55, 3), disk_pack_2d(40, 0.5, 1)
    solves = [(a, "fp64", {}), (b, "fp64", {}), (a, "fp32", {}), (c, "fp32", {}),
              (a, "fp64", dict(force=3e-6)), (a, "fp64", dict(tau_lb=0.9)),
              (a, "fp64", dict(magic=0.25)), (a, "fp64", dict(nit=250)), (b, "fp64", dict(tol=1e-2))]
    kinds = [(s, t) for s in solves for t in ("0", "1")]

    def solve(kind, ctx):
        (g, precision, kw), table = kind
        monkeypatch.setenv("PRT_NBR_TABLE", table)
        return flow(g, precision, ctx=ctx, **kw)

    def alone(kind):
        ctx = _lib.Context(0)
        try:
            return solve(kind, ctx)
        finally:
            ctx.close()

    want = [alone(k) for k in kinds]
    ctx = _lib.Context(0)
    try:
        for _ in range(2):
            for k, w in zip(kinds, want):
                same(solve(k, ctx), w)
    finally:
        ctx.close()


@pytest.mark.parametrize("precision", ["fp64", "fp32", "fp32f", "fp16"])
@pytest.mark.parametrize("taus", [(0.8, 0.8), (0.8, 0.9)], ids=["shared", "own"])
def test_batched_flow_from_packed_and_plain_tables(monkeypatch, precision, taus):
    """A batch whose jobs have no plain table reads the packed ones; constants
    shared by the jobs or each job's own."""
    from prtlb_gpu import random_pack
    from prtlb_gpu.batch import Request, solve_batch
    grids = [random_pack((21, 18, 23), 0.5, 2.0, 3.5, seed=1), random_pack((8, 40, 33), 0.7, 2.0, 3.5, seed=2),
             random_pack((44, 37), 0.6, 2.0, 4.0, seed=3), np.full((5, 4, 8), 2, np.uint8)]
    grids[1][::2, ::3] = 0  # gaps wider than a packed byte: warps that go to the maps
    grids += [g.copy() for g in grids[:2]]
    tau = [taus[i % 2] for i in range(len(grids))]
    tau[4] = tau[5] = taus[1]
    want = [flow(g, precision, nit=333, tol=0.0, tau_lb=t)[0] for g, t in zip(grids, tau)]
    for table in ("0", "1"):
        monkeypatch.setenv("PRT_NBR_TABLE", table)
        got = solve_batch([Request(g, flow=dict(nit=333, tol=0.0, precision=precision, tau_lb=t),
                                   keep_velocity=True) for g, t in zip(grids, tau)], quiet=True)
        for r, w in zip(got, want):
            assert r.error is None, r.error
            assert np.array_equal(r.vel, w)
