"""What calls of one process share: a limit that belongs to a kernel."""

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
