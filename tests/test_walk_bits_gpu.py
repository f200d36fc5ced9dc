"""The walk on bit masks inside one cluster against the walk by launches
(PRT_CLUSTER=0) and, where it is quick, the oracle: rows around whole words of
32 voxels, fewer rows than blocks, axes of one voxel, every seed axis and
both ends, pore that is not reached, no pore, a path longer than a vote's
levels, and the largest grid one cluster takes with one that it does not."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def grid(name):
    rng = np.random.default_rng(7)
    if name == "empty":
        return np.zeros((5, 6, 7), np.uint8)
    if name == "serpentine":
        g = np.zeros((40, 61), np.uint8)
        g[:, ::2] = 2
        g[-1, 1::4] = 2
        g[0, 3::4] = 2
        return g
    shape = {"z31": (9, 8, 31), "z32": (9, 8, 32), "z33": (7, 11, 33), "z65": (5, 3, 65),
             "thin_x": (1, 20, 40), "thin_y": (33, 1, 70), "z1": (19, 21, 1), "few_rows": (3, 3, 100),
             "flat": (70, 90), "row": (1, 50), "column": (50, 1)}[name]
    return np.where(rng.random(shape) < 0.66, 2, 0).astype(np.uint8)


GRIDS = ["z31", "z32", "z33", "z65", "thin_x", "thin_y", "z1", "few_rows", "flat", "row", "column",
         "empty", "serpentine"]


def both_ways(monkeypatch, g, axis, plane):
    from prtlb_gpu import prep
    found = []
    for on in ("0", "1"):
        monkeypatch.setenv("PRT_CLUSTER", on)
        found.append(prep.walk_from_plane(g, 2, axis, plane))
    assert found[0][1:] == found[1][1:]
    assert np.array_equal(found[0][0], found[1][0])
    return found[1]


@pytest.mark.parametrize("name", GRIDS)
def test_bits_give_the_steps_of_the_launches(monkeypatch, name):
    from oracle.prep_oracle import geodesic_steps
    g = grid(name)
    for axis in range(g.ndim):
        for plane in (0, -1):
            both_ways(monkeypatch, g, axis, plane)
        steps = both_ways(monkeypatch, g, axis, 0)[0]
        want = geodesic_steps(g == 2, axis)
        assert np.array_equal(steps >= 0, ~np.isnan(want))
        assert np.array_equal(steps[steps >= 0], want[steps >= 0].astype(np.int32))


@pytest.mark.parametrize("shape", [(64, 256, 512), (64, 256, 513)])
def test_largest_grid_of_one_cluster_and_the_next(monkeypatch, shape):
    """16 words a row and 1024 rows a block fill the masks; one voxel more
    along z is a seventeenth word and takes the launches."""
    g = np.where(np.random.default_rng(1).random(shape) < 0.8, 2, 0).astype(np.uint8)
    steps, reached, pore = both_ways(monkeypatch, g, 0, 0)
    assert pore == int((g == 2).sum()) and reached == int((steps >= 0).sum())
