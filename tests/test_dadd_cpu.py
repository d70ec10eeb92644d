"""The integer-pipe addition of positive numbers and products by 3, 5, 7 and 11
(dadd_pos, dmul_small in amrsolver_gb300/csrc/ddiv.cuh) on the host against the
host's operations, bit for bit."""
import os
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))


@pytest.mark.parametrize("seed", [21, 22])
def test_dadd_pos(tmp_path, seed):
    exe = str(tmp_path / "dadd_check")
    subprocess.check_call(["g++", "-O2", "-std=c++17", "-o", exe, os.path.join(HERE, "cpp", "dadd_check.cpp")])
    r = subprocess.run([exe, "10000000", str(seed)], capture_output=True, text=True)
    assert r.returncode == 0 and "mismatches 0 checked" in r.stdout, r.stdout
