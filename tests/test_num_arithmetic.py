"""Num expressions of spd_soft.cuh: a result flagged as in range has the IEEE
bits (host and GPU)."""
import os
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(os.path.dirname(HERE), "spd_gb300", "csrc")


@pytest.mark.parametrize("where", ["host", pytest.param("gpu", marks=pytest.mark.gpu)])
def test_num_results_in_range_are_ieee(tmp_path, where):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(nvcc):
        pytest.skip("nvcc not available")
    exe = str(tmp_path / "host_num_check")
    subprocess.run([nvcc, "-std=c++17", "-O1", "--fmad=false", "-gencode", "arch=compute_103a,code=sm_103a",
                    "-I", CSRC, os.path.join(HERE, "host_num_check.cu"), "-o", exe], check=True)
    out = subprocess.run([exe, where], capture_output=True, text=True)
    assert out.returncode == 0, out.stdout + out.stderr
