"""The forms of a flow step, chosen by how many blocks the device holds at once:
the same field bit for bit on both sides of each line as from the batch's
kernel, whose form does not depend on the size.  Slot counts around the lines
of a device of 148 SMs; any device holds some of each."""

import contextlib
import io

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def grid(plane, slots, seed=0):
    """Rows of `plane` until `slots` pore voxels and some rock fit."""
    n = int(np.prod(plane))
    rows = -(-(slots + slots // 20 + 1) // n)
    g = np.full(rows * n, 2, np.uint8)
    g[np.random.default_rng(seed).permutation(g.size)[:g.size - slots]] = 0
    assert (g == 2).sum() == slots
    return g.reshape((rows,) + plane)


LINES = ([("fp64", (40, 48), 128 * b + d) for b in (592, 740) for d in (0, 1)]
         + [("fp64", (330,), 128 * b + d) for b in (1036, 1332) for d in (0, 1)]
         + [(p, (330,), 128 * b + d) for p in ("fp32f", "fp16") for b in (1332, 1480)
            for d in (0, 1)])


@pytest.mark.parametrize("precision,plane,slots", LINES)
def test_forms_give_the_batch_kernels_field(precision, plane, slots):
    from prtlb_gpu import stokes_d2q9, stokes_d3q19
    from prtlb_gpu.batch import Request, solve_batch
    g = grid(plane, slots)
    info = {}
    with contextlib.redirect_stdout(io.StringIO()):
        v = (stokes_d3q19 if g.ndim == 3 else stokes_d2q9)(g, nit=103, tol=1e-12, info=info,
                                                           precision=precision)
    r, = solve_batch([Request(g, flow=dict(nit=103, tol=1e-12, precision=precision),
                              keep_velocity=True)], quiet=True)
    assert r.error is None, r.error
    assert np.array_equal(v, r.vel), float(np.abs(v - r.vel).max())
    assert info["flow_change"] == r.flow_info["flow_change"]
