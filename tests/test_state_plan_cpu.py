"""How the state scans are spread over the SMs: one host rule picks segments of the sequence or even shares of chunks."""
import os
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))


def test_segments_and_even_shares_exclude_each_other(tmp_path):
    """Rule and block walks (csrc/state_plan.h) compiled for the host: 1-2000 units x 1-1200 chunks never choose both, and
    the replayed walks of all blocks visit every chunk once, keep their hand-over slots inside the array, and end every unit."""
    cxx = shutil.which("g++")
    if cxx is None:
        pytest.skip("no host compiler")
    exe = str(tmp_path / "state_plan_check")
    subprocess.run([cxx, "-std=c++17", "-O2", "-Wall", os.path.join(HERE, "cpp", "state_plan_check.cpp"), "-o", exe], check=True)
    r = subprocess.run([exe], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout
