"""Fused build: the first Picard iteration rounds a sum once per term."""
import os
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(os.path.dirname(HERE), "spd_gb300", "csrc")


def test_first_picard_iteration_of_the_fused_build_fuses_its_terms(tmp_path):
    cxx = shutil.which("g++")
    if cxx is None:
        pytest.skip("g++ not available")
    exe = str(tmp_path / "host_picard_check")
    # no contraction by the compiler: only the fused multiply-adds in the source
    subprocess.run([cxx, "-std=c++17", "-O1", "-w", "-ffp-contract=off", "-DSPD_FUSED", "-I", HERE, "-I", CSRC,
                    os.path.join(HERE, "host_picard_check.cpp"), "-o", exe], check=True)
    out = subprocess.run([exe], capture_output=True, text=True)
    assert out.returncode == 0, out.stdout + out.stderr
