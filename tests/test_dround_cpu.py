"""Quotients and roots next to a midpoint between two doubles (ddiv_core and dsqrt_core in
amrsolver_gb300/csrc/ddiv.cuh) on the host against the host's operations, bit for bit."""
import os
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))


@pytest.mark.parametrize("seed", [31, 32])
def test_undecided_roundings(tmp_path, seed):
    exe = str(tmp_path / "dround_check")
    subprocess.check_call(["g++", "-O2", "-std=c++17", "-o", exe, os.path.join(HERE, "cpp", "dround_check.cpp")])
    r = subprocess.run([exe, "3000000", str(seed)], capture_output=True, text=True)
    assert r.returncode == 0 and "mismatches 0 checked" in r.stdout, r.stdout
