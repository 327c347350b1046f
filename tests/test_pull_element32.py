"""The 32-bit addresses of a batch's special cells (d3q19.cuh: pull_element<I, int>), on the CPU: the 64-bit ones
up to the 2^30 cells a batch case can have, without a signed overflow on the way.  Whole numbers, so equal."""
import os
import shutil
import subprocess

import pytest

SOURCE = os.path.join(os.path.dirname(os.path.abspath(__file__)), "native", "pull_element32_check.cu")


@pytest.mark.skipif(shutil.which("nvcc") is None, reason="needs nvcc (host compilation only)")
def test_32_bit_addresses_are_the_64_bit_ones(tmp_path):
    exe = tmp_path / "pull32"
    subprocess.check_call(["nvcc", "-O1", "-std=c++17", "-Xcompiler",
                           "-fsanitize=signed-integer-overflow,-fno-sanitize-recover=signed-integer-overflow",
                           SOURCE, "-o", str(exe)])
    run = subprocess.run([str(exe)], capture_output=True, text=True)
    assert run.returncode == 0 and run.stdout.split() == [str(4 * 4000 * 19), "0"], run.stdout + run.stderr
