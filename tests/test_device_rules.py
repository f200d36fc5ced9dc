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
