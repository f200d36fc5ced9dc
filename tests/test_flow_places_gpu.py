"""Where an iteration finds its far places: the plain table, and the packed
table with the maps behind it, give the same places, so the same field bit for bit, on grids
that reach their edges -- axes of 1, 2 and 3 voxels (the periodic neighbour is
the voxel itself, or the same on both sides), warps that cross the ends of
the grid or gaps wider than a packed byte, slot counts around a warp and a
block, no rock, isolated pore voxels.  float64 is held to the NumPy oracle:
the field is stored as float32, so 1e-6 of its maximum is a few of its
roundings."""

import contextlib
import ctypes
import io

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def grid(name):
    rng = np.random.default_rng(len(name))
    if name == "no_rock":
        g = np.full((5, 4, 8), 2, np.uint8)
    elif name == "one_voxel":
        g = np.zeros((3, 3, 3), np.uint8)
        g[1, 1, 1] = 2
    elif name == "isolated":  # every place but the own one is a link
        g = np.zeros((12, 12, 12), np.uint8)
        g[::3, ::3, ::3] = 2
    elif name == "row_of_33":
        g = np.full((1, 1, 33), 2, np.uint8)
    elif name == "thin_y":
        g = np.where(rng.random((17, 1, 23)) < 0.7, 2, 0).astype(np.uint8)
    elif name == "two_by_three":
        g = np.where(rng.random((2, 3, 45)) < 0.6, 2, 0).astype(np.uint8)
    elif name == "wide_gap":  # open and nearly closed planes: far slots > 255 apart
        g = np.full((8, 40, 40), 2, np.uint8)
        g[::2] = 0
        g[::2, 7, ::5] = 2
    elif name == "long_rows":  # rows of more than 255 slots
        g = np.where(rng.random((4, 5, 700)) < 0.8, 2, 0).astype(np.uint8)
    elif name == "site3d":
        g = np.where(rng.random((19, 23, 21)) < 0.55, 2, 0).astype(np.uint8)
    elif name == "line2d":
        g = np.full((1, 129), 2, np.uint8)
        g[0, ::7] = 0
    else:
        g = np.where(rng.random((37, 301)) < 0.75, 2, 0).astype(np.uint8)
    return g


# voxels around what one cluster takes: one block, all 16, the most and one more
EDGES = [("fp64", (1, 1, 128)), ("fp64", (8, 16, 16)), ("fp64", (16, 16, 32)), ("fp64", (16, 16, 33)),
         ("fp32", (16, 16, 32)), ("fp32f", (16, 32, 20)), ("fp16", (10, 32, 32)), ("fp64", (128, 128)),
         ("fp32f", (129, 127)), ("fp64", (128, 129))]


GRIDS = ["no_rock", "one_voxel", "isolated", "row_of_33", "thin_y", "two_by_three", "wide_gap",
         "long_rows", "site3d", "line2d", "site2d"]


def solve(g, precision, nit):
    from prtlb_gpu import stokes_d2q9, stokes_d3q19
    with contextlib.redirect_stdout(io.StringIO()):
        return (stokes_d3q19 if g.ndim == 3 else stokes_d2q9)(g, nit=nit, tol=0.0,
                                                              precision=precision)


def without_allocation(g, precision, nit):
    """The field of prt_flow_noalloc, whose tables lie in its own scratch."""
    import torch
    from prtlb_gpu import _lib
    from prtlb_gpu.flow import flow_params
    g8, p = flow_params(g, g.ndim, "flow", nit, 2e-6, 0.8, 3.0 / 16.0, 0.0, precision)
    d_mat = torch.from_numpy(g8).cuda()
    d_vel = torch.empty((3,) + g.shape, dtype=torch.float32, device="cuda")
    torch.cuda.synchronize()
    rc = _lib.lib().prt_flow_noalloc(ctypes.c_void_p(d_mat.data_ptr()), ctypes.byref(p),
                                     ctypes.c_void_p(d_vel.data_ptr()), None, None)
    assert rc == 0, _lib.lib().prt_last_error(None)
    return d_vel.cpu().numpy()


@pytest.mark.parametrize("precision", ["fp64", "fp32", "fp32f", "fp16"])
@pytest.mark.parametrize("name", GRIDS)
def test_places_from_tables_and_maps_are_the_same(monkeypatch, name, precision):
    g = grid(name)
    nit = 53
    monkeypatch.setenv("PRT_CLUSTER", "0")
    monkeypatch.setenv("PRT_NBR_TABLE", "1")
    plain = solve(g, precision, nit)
    monkeypatch.setenv("PRT_NBR_TABLE", "0")
    packed = solve(g, precision, nit)
    assert np.array_equal(plain, packed)
    assert np.array_equal(plain, without_allocation(g, precision, nit))
    # the loop inside one cluster, whose blocks' places lie in one another's
    # shared memory
    monkeypatch.setenv("PRT_CLUSTER", "1")
    assert np.array_equal(plain, solve(g, precision, nit))
    if precision == "fp64":
        from oracle.prtlb_oracle import stokes
        ref = stokes(g, nit=nit, tol=0.0)
        assert np.abs(plain - ref).max() <= 1e-6 * np.abs(ref).max()


@pytest.mark.parametrize("tol", [0.0, 1e-3])
@pytest.mark.parametrize("precision,shape", EDGES)
def test_cluster_loop_is_the_launches(monkeypatch, precision, shape, tol):
    """Fields and iteration counts of the loop inside one cluster against the
    launches, at a count that is no multiple of the check interval and with
    the stop rule."""
    from prtlb_gpu import stokes_d2q9, stokes_d3q19
    g = np.full(shape, 2, np.uint8)
    g.reshape(-1)[5::97] = 0
    found = []
    for on in ("0", "1"):
        monkeypatch.setenv("PRT_CLUSTER", on)
        info = {}
        with contextlib.redirect_stdout(io.StringIO()):
            v = (stokes_d3q19 if g.ndim == 3 else stokes_d2q9)(g, nit=333, tol=tol, info=info,
                                                               precision=precision)
        found.append((v, info["flow_iters"], info["flow_change"], info["permeability"]))
    assert np.array_equal(found[0][0], found[1][0])
    assert found[0][1:] == found[1][1:]
