"""Euler maps and Riemann solvers of the step's kernels against plain FP64
arithmetic at the ends of the integer-pipe products' range (host and GPU)."""
import os
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(os.path.dirname(HERE), "spd_gb300", "csrc")


@pytest.mark.parametrize("where", ["host", pytest.param("gpu", marks=pytest.mark.gpu)])
def test_maps_equal_plain_arithmetic_at_the_ends_of_the_range(tmp_path, where):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(nvcc):
        pytest.skip("nvcc not available")
    exe = str(tmp_path / "host_maps_check")
    # no contraction on the host either (aarch64 has a fused multiply-add)
    subprocess.run([nvcc, "-std=c++17", "-O1", "--fmad=false", "-Xcompiler", "-ffp-contract=off", "-gencode",
                    "arch=compute_103a,code=sm_103a", "-I", CSRC, os.path.join(HERE, "host_maps_check.cu"), "-o", exe],
                   check=True)
    out = subprocess.run([exe, where], capture_output=True, text=True)
    assert out.returncode == 0, out.stdout + out.stderr
