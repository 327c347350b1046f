"""Eight channels a thread (channels.cuh), on the CPU: the vector accesses fall on the arrays in memory only,
so a local array of plain floats may lie at any 4-byte boundary."""
import os
import shutil
import subprocess

import pytest

SOURCE = os.path.join(os.path.dirname(os.path.abspath(__file__)), "native", "channels_check.cu")


@pytest.mark.skipif(shutil.which("nvcc") is None, reason="needs nvcc (host compilation only)")
def test_local_arrays_need_no_alignment(tmp_path):
    exe = tmp_path / "channels"
    subprocess.check_call(["nvcc", "-O1", "-std=c++17", "-Xcompiler", "-fsanitize=alignment,-fno-sanitize-recover=alignment",
                           SOURCE, "-o", str(exe)])
    run = subprocess.run([str(exe)], capture_output=True, text=True)
    assert run.returncode == 0 and run.stdout.split() == ["0"], run.stdout + run.stderr
