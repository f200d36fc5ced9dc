"""Rules of the library's host code that no result shows, on the CPU: a small
program that includes the headers states them."""

import os
import shutil
import subprocess

import pytest

from conftest import PKG, ROOT

pytestmark = pytest.mark.skipif(shutil.which("nvcc") is None, reason="needs nvcc")


def holds(tmp_path, body):
    src, exe = tmp_path / "rule.cu", tmp_path / "rule"
    src.write_text('#include <cstdlib>\n#include "prt_internal.h"\nusing namespace prt;\n'
                   "int main() {\n%s\n}\n" % body)
    subprocess.run(["nvcc", "-gencode", "arch=compute_100a,code=sm_100a", "-std=c++17",
                    "-I", os.path.join(PKG, "csrc"), "-I", os.path.join(ROOT, "include"),
                    "-o", str(exe), str(src)], check=True)
    return subprocess.run([str(exe)], timeout=60).returncode == 0


def test_forced_plain_tables_hold_for_large_batches(tmp_path):
    assert holds(tmp_path, """
    const long long l2 = 126ll << 20;
    unsetenv("PRT_NBR_TABLE");
    bool good = batch_use_nbr(l2 / 4 * 3, l2) && !batch_use_nbr(l2, l2);
    setenv("PRT_NBR_TABLE", "1", 1);
    good = good && batch_use_nbr(l2, l2) && batch_use_nbr(100 * l2, l2);
    setenv("PRT_NBR_TABLE", "0", 1);  // such solves have no plain table to read
    return good && !batch_use_nbr(l2, l2) ? 0 : 1;""")


def test_table_places_do_not_wrap(tmp_path):
    """Three axes of more than 1.4e9 solute voxels exceed 32 bits: such runs have
    neighbour places, whose tables are counted in 64."""
    assert holds(tmp_path, """
    const long long nm = 2147483000ll;  // the most solute voxels a grid may have, nearly
    const unsigned k = 2147482999u;
    const long long last = (1ll << 32) / 3;  // the most with distances in 3D
    return !adr_use_near(100, 3, nm) && axis_place<true>(2, k, nm) == 3ull * nm - 1 &&
           adr_use_near(65535, 3, last) && !adr_use_near(65535, 3, last + 1) &&
           axis_place<false>(2, (unsigned)last - 1, last) == 3ull * last - 1 &&
           adr_use_near(65535, 2, nm) && axis_place<false>(1, k, nm) == 2ull * nm - 1 &&
           !adr_use_near(65536, 2, 100) ? 0 : 1;""")
