"""Admission's estimate against the transport's buffers, added up from their
definitions: rows of the state with the inlet plane's values behind them, and
neighbour places where distances need more than 16 bits."""

import numpy as np
import pytest


def transport_bytes(g, ns, slots, limit):
    """The device buffers of a transport run, as prt_adr_stage, prt_adr_begin,
    prt_adr_run and prt_adr_fetch make them."""
    n, nd = g.size, g.ndim
    m = g == 2
    nm, n0 = int(m.sum()), int(m[0].sum())
    order = np.cumsum(m.reshape(-1)).reshape(g.shape) - 1
    reach = 0
    for axis in range(nd):
        for d in (1, 2):
            lo = tuple(slice(0, -d) if a == axis else slice(None) for a in range(nd))
            hi = tuple(slice(d, None) if a == axis else slice(None) for a in range(nd))
            both = m[lo] & m[hi]
            if both.any():
                reach = max(reach, int((order[hi] - order[lo])[both].max()))
    near = 8 if reach <= 0xffff else 16
    ms = (nm + n0 + 31) // 32 * 32
    per_grid = n * (1 + 12) + n * (4 + 1 + 4) + 4 * n * ns
    per_solute = nm * (4 + near * nd + 8 * nd + 4)
    leaves = nm // 65  # numpy's pairwise leaves hold more than 64 values of a large row
    tree = leaves * (4 + 4 + 4 + 4) + 2 * leaves * 8 * 4
    return per_grid + per_solute + tree + 2 * 4 * ns * ms + 4 * nm * ns * slots + 4 * (limit + 1)


@pytest.mark.parametrize("shape", [(3, 190, 190), (4, 1000, 1000), (400, 16, 16), (2, 1000000), (64, 64)])
@pytest.mark.parametrize("ns", [1, 4])
def test_footprint_covers_the_transport(shape, ns):
    from prtlb_gpu.batch import Request
    from prtlb_gpu.serve import footprint, ladder_slots
    g = np.full(shape, 2, np.uint8)  # nothing to spare in what is counted by the voxel
    limit = 1
    r = Request(g, flow=dict(nit=1, precision="fp16"),
                adr=dict(pe=1.0, da=1.0, n_t=2, n_species=ns, steps=limit))
    assert footprint(r) >= transport_bytes(g, ns, ladder_slots(limit, 1.12), limit)
