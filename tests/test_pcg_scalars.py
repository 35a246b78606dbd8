"""The recurrence scalars of the persistent PCG, compiled for the host."""

import os
import shutil
import subprocess

import pytest


def test_pcg_scalars_keep_fp64_for_vectors_of_both_types(tmp_path):
    """tests/native/pcg_scalars_check.cpp: r.z, r.r and the stopping limit keep their 53 bits and FP64's range, and the
    quotients are FP64 quotients rounded once; ends, breakdowns and NaN give their statuses."""
    gxx = shutil.which("g++")
    if gxx is None:
        pytest.skip("no C++ compiler")
    exe = str(tmp_path / "pcg_scalars_check")
    source = os.path.join(os.path.dirname(os.path.abspath(__file__)), "native", "pcg_scalars_check.cpp")
    subprocess.run([gxx, "-O2", "-std=c++17", "-o", exe, source], check=True)
    out = subprocess.run([exe], capture_output=True, text=True)
    assert out.returncode == 0 and "failures 0" in out.stdout, out.stdout + out.stderr
