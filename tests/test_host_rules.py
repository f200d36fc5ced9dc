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
