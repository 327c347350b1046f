"""Addresses of the special cells' pull (d3q19.cuh: pull_element), on the CPU: lattices below and above
2^30 and 2^31 cells, every direction at walls, x ends, under the lid and inside, against the rule in
coordinates and 64 bits.  Whole numbers, so equal."""
import os
import shutil
import subprocess

import pytest

SOURCE = os.path.join(os.path.dirname(os.path.abspath(__file__)), "native", "pull_element_check.cu")


@pytest.mark.skipif(shutil.which("nvcc") is None, reason="needs nvcc (host compilation only)")
def test_pull_element_is_the_pull_rule(tmp_path):
    exe = tmp_path / "pull"
    subprocess.check_call(["nvcc", "-O2", "-std=c++17", SOURCE, "-o", str(exe)])
    compared, differ, outside = map(int, subprocess.run([str(exe)], capture_output=True, text=True, check=True).stdout.split())
    assert (compared, differ, outside) == (6 * 4000 * 19, 0, 0)
