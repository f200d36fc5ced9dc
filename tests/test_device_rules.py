"""Rules of the device code that no result shows reliably, read from its source."""

import glob
import os
import re

from conftest import PKG

SOURCES = sorted(glob.glob(os.path.join(PKG, "csrc", "*.cu*")))


def code(path):
    """The file without its comments."""
    with open(path) as f:
        return re.sub(r"//[^\n]*|/\*.*?\*/", "", f.read(), flags=re.S)


def test_no_read_only_load_by_hand():
    """ld.global.nc asks that nothing writes the data while the reading kernel
    is resident.  Step launches overlap, and what they load by hand is the
    state, which the step before writes; tables go through __ldg."""
    assert SOURCES
    for path in SOURCES:
        assert ".nc." not in code(path), path


def test_aligned_cluster_barriers_follow_a_warp_barrier():
    """The .aligned forms need a converged warp, which code behind a divergent
    branch does not promise."""
    found = 0
    for path in SOURCES:
        for before in re.split(r"asm volatile\(\s*\"barrier\.cluster\.\S+\.aligned", code(path))[:-1]:
            assert before.rstrip().endswith("__syncwarp();"), path
            found += 1
    assert found
