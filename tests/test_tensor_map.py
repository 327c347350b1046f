"""The driver's tensor-map encoder (tensor_map.cuh: encode_tiled), on the CPU with a slow driver: threads
that need it for the first time together all get it, none a NULL while another is still asking."""
import os
import shutil
import subprocess

import pytest

SOURCE = os.path.join(os.path.dirname(os.path.abspath(__file__)), "native", "encode_tiled_check.cpp")


@pytest.mark.skipif(shutil.which("nvcc") is None, reason="needs the CUDA headers")
def test_every_thread_gets_the_encoder(tmp_path):
    exe = tmp_path / "encode"
    include = os.path.join(os.path.dirname(os.path.dirname(os.path.realpath(shutil.which("nvcc")))), "include")
    subprocess.check_call(["g++", "-O2", "-std=c++17", "-pthread", "-I", include, SOURCE, "-o", str(exe)])
    assert subprocess.run([str(exe)], capture_output=True, text=True, check=True).stdout.split() == ["8"]
