"""The compact transport state against the NumPy oracle, bit for bit, where its
tables can go wrong: axes of 1, 2 and 3 voxels, rock on and off the inlet
plane, an all-pore grid, one voxel, warps and blocks that end mid-row, fed,
unfed and immobile chemicals on the inlet plane, a surface reaction -- with
16-bit neighbour distances and with neighbour places (PRT_ADR_WIDE=1), by
launches and inside one cluster (PRT_CLUSTER), alone and in a batch; and the same fields on a grid whose distances exceed 16 bits
(so that only the places can hold them) as on two halves of it."""

import contextlib
import io

import numpy as np
import pytest

from golden.fields import integer_velocity

pytestmark = pytest.mark.gpu


def grid(name):
    rng = np.random.default_rng(3)
    shapes = {"thin_x": (1, 9, 14), "two_x": (2, 7, 13), "three_x": (3, 6, 11),
              "thin_y": (17, 1, 12), "site3d": (13, 11, 17), "site2d": (29, 23),
              "line2d": (41, 1)}
    if name == "all_pore":
        return np.full((6, 5, 8), 2, np.uint8)
    if name == "one_voxel":
        g = np.zeros((4, 3, 3), np.uint8)
        g[2, 1, 1] = 2
        return g
    if name == "no_inlet":
        g = np.where(rng.random((9, 8, 7)) < 0.7, 2, 0).astype(np.uint8)
        g[0] = 0
        return g
    return np.where(rng.random(shapes[name]) < 0.72, 2, 0).astype(np.uint8)


GRIDS = ["thin_x", "two_x", "three_x", "thin_y", "site3d", "site2d", "line2d", "all_pore",
         "one_voxel", "no_inlet"]


def chemistry(kind):
    from prtlb_gpu import Chemistry, default_chemistry, monod_chemistry
    if kind == "monod":
        return monod_chemistry(0.5), 1, 0.0
    if kind == "default4":
        return default_chemistry(4), 4, 0.0
    # a mobile product that is not fed, and a surface-only abiotic reaction
    nan = np.float32(np.nan)
    return Chemistry(names=["A", "B", "P"], inlet=[1.0, 0.5, nan], c_init=[0.1, 0.0, 0.2],
                     d_rel=[1.0, 0.7, 1.3], immobile=[False, False, False], ks_donor=0.3,
                     abiotic_surface_only=True, abiotic_index=1, abiotic_product_index=2), 3, 2.0


def arguments(g, kind, steps):
    chem, ns, da_abio = chemistry(kind)
    return dict(pe=8.0, da=1.5, n_t=4, n_species=ns, steps=steps, chem=chem, da_abio=da_abio)


def solve(g, v, kw):
    from prtlb_gpu import solve_adr
    with contextlib.redirect_stdout(io.StringIO()):
        return solve_adr(g, v, **kw)


@pytest.mark.parametrize("kind", ["monod", "default4", "surface3"])
@pytest.mark.parametrize("name", GRIDS)
def test_steps_equal_the_oracle(monkeypatch, name, kind):
    from oracle.prtlb_oracle import solve_adr as reference
    g = grid(name)
    v = integer_velocity(g)
    kw = arguments(g, kind, 37)
    with contextlib.redirect_stdout(io.StringIO()):
        want, _ = reference(g, v, kw["pe"], kw["da"], kw["n_t"], n_species=kw["n_species"],
                            steps=kw["steps"], chem=kw["chem"], da_abio=kw["da_abio"])
    for wide, cluster in (("0", "0"), ("1", "0"), ("0", "1"), ("1", "1")):
        monkeypatch.setenv("PRT_ADR_WIDE", wide)
        monkeypatch.setenv("PRT_CLUSTER", cluster)
        out, _ = solve(g, v, kw)
        assert np.array_equal(out, want), (wide, cluster, float(np.abs(out - want).max()))


def test_wide_neighbours_in_a_batch(monkeypatch):
    from prtlb_gpu.batch import Request, solve_batch
    from prtlb_gpu import sphere_pack_3d
    reqs = [Request(sphere_pack_3d(n, 0.5, n), flow=dict(nit=100, tol=0.0, precision="fp32"),
                    adr=arguments(None, kind, 220))
            for n, kind in ((20, "monod"), (24, "default4"), (28, "surface3"))]
    monkeypatch.setenv("PRT_ADR_WIDE", "0")
    near = solve_batch(reqs, quiet=True)
    monkeypatch.setenv("PRT_ADR_WIDE", "1")
    wide = solve_batch(reqs, quiet=True)
    for a, b in zip(near, wide):
        assert a.error is None and b.error is None
        assert np.array_equal(a.out, b.out)


def test_distances_beyond_16_bits():
    """Two planes of more than 32768 solute voxels: the far neighbours along x
    are more than 65535 voxels apart.  The flow is along x only and the grid
    is two equal halves side by side along y with rock between, so each half
    is the smaller grid's solve, whose distances fit 16 bits."""
    half = np.full((5, 128, 140), 2, np.uint8)
    half[:, 0] = half[:, -1] = 0
    rng = np.random.default_rng(5)
    half[:, 1:-1][rng.random((5, 126, 140)) < 0.05] = 0
    both = np.concatenate([half, half], axis=1)
    v1 = integer_velocity(half)
    v1[1:] = 0.0
    v2 = np.concatenate([v1, v1], axis=2)
    assert 2 * int((both[0] == 2).sum()) > 65535 > 2 * int((half[0] == 2).sum())
    kw = arguments(half, "monod", 25)
    a, _ = solve(half, v1, kw)
    b, _ = solve(both, v2, kw)
    assert np.array_equal(b[:, :, :, :128], a) and np.array_equal(b[:, :, :, 128:], a)


# solute voxels around what one cluster takes: one block, all 16, the most and more
@pytest.mark.parametrize("kind", ["monod", "default4", "surface3"])
@pytest.mark.parametrize("shape", [(4, 4, 8), (16, 16, 9), (20, 16, 32), (20, 16, 33), (80, 128)])
def test_cluster_loop_is_the_launches(monkeypatch, shape, kind):
    """Snapshots, times, stop step and progress records of the loop inside one
    cluster against the launches, under the stop rule with its pauses for the
    callback, and for a step count that is no multiple of the check interval."""
    g = np.full(shape, 2, np.uint8)
    g.reshape(-1)[37::61] = 0
    g[0, 0] = 2
    v = integer_velocity(g)
    for steps, most in ((None, 2500), (271, 0)):
        found = []
        for cluster in ("0", "1"):
            monkeypatch.setenv("PRT_CLUSTER", cluster)
            seen, info = [], {}
            kw = arguments(g, kind, steps)
            out, t = solve(g, v, dict(kw, max_steps=most or 100000, info=info,
                                      on_progress=lambda *a: seen.append(a)))
            found.append((out, t, info["steps"], info["ladder"], seen))
        assert np.array_equal(found[0][0], found[1][0])
        assert np.array_equal(found[0][1], found[1][1])
        assert found[0][2:] == found[1][2:]


def test_long_check_intervals_run_in_segments(monkeypatch):
    """At a low Peclet number the check interval (here 1 500 steps) exceeds a
    graph body, so a check follows several segments; the stop step, the
    progress records and the fields are those of direct launches, of one
    cluster, and of the oracle's step rule."""
    from oracle.prtlb_oracle import solve_adr as reference
    g = np.full((24, 20), 2, np.uint8)
    g[5::7, ::3] = 0
    v = integer_velocity(g)
    kw = dict(pe=0.16, da=2.0, n_t=3, n_species=1, max_steps=3100, chem=chemistry("monod")[0])
    with contextlib.redirect_stdout(io.StringIO()):
        said = []
        want, _ = reference(g, v, kw["pe"], kw["da"], 3, n_species=1, max_steps=3100,
                            chem=kw["chem"], on_progress=lambda *a: said.append(a))
    assert len(said) == 2 and said[0][0] > 1000
    for cluster, graphs in (("0", "1"), ("0", "0"), ("1", "1")):
        monkeypatch.setenv("PRT_CLUSTER", cluster)
        monkeypatch.setenv("PRT_GRAPHS", graphs)
        seen = []
        out, _ = solve(g, v, dict(kw, on_progress=lambda *a: seen.append(a)))
        assert np.array_equal(out, want)
        assert [a[0] for a in seen] == [a[0] for a in said]
