"""The viscous kernels stay within the arrays that the context allocates: their
bodies run on the CPU on arrays that end at an inaccessible page."""
import os
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(os.path.dirname(HERE), "spd_gb300", "csrc")


def test_viscous_kernels_stay_within_their_arrays(tmp_path):
    cxx = shutil.which("g++")
    if cxx is None:
        pytest.skip("g++ not available")
    exe = str(tmp_path / "host_visc_check")
    # -O0: every load in the source is made
    subprocess.run([cxx, "-std=c++17", "-O0", "-w", "-I", HERE, "-I", CSRC, os.path.join(HERE, "host_visc_check.cpp"),
                    "-o", exe], check=True)
    out = subprocess.run([exe], capture_output=True, text=True)
    assert out.returncode == 0, f"exit status {out.returncode}: {out.stdout}{out.stderr}"
