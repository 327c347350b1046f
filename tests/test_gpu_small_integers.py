"""The wall function's tabulated and corrected operations on the device (d3q19.cuh: div_small, sqrt_small,
int_double), compiled as the library is: the bits of p / n, sqrt(k) and (double)k (needs a B200)."""
import os
import subprocess

import pytest

SOURCE = os.path.join(os.path.dirname(os.path.abspath(__file__)), "native", "small_integers_check.cu")


@pytest.mark.gpu
def test_small_integer_operations_round_as_the_general_ones(tmp_path):
    from water_flow_simulation_b200 import _native as nat
    exe = tmp_path / "small"
    flags = [f for f in nat.NVCC_FLAGS if f not in ("-Xcompiler", "-fPIC", "-shared")]
    subprocess.check_call(["nvcc", *flags, SOURCE, "-o", str(exe)])
    run = subprocess.run([str(exe)], capture_output=True, text=True)
    assert run.returncode == 0 and run.stdout.split() == [str(75 * 20000 + 13 + 8193), "0"], run.stdout + run.stderr
