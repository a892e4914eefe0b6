"""How the state scans are spread over the SMs: one host rule, and the order in which a block walks its chunks."""
import os
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))


def test_state_plan_and_walks(tmp_path):
    """Rule and block walks (csrc/state_plan.h) compiled for the host: even shares only where a share is longer than a unit (1-2000
    units x 1-1200 chunks), and the replayed walks of all blocks visit every chunk once and in order, keep their hand-over slots
    inside the array, and end every unit."""
    cxx = shutil.which("g++")
    if cxx is None:
        pytest.skip("no host compiler")
    exe = str(tmp_path / "state_plan_check")
    subprocess.run([cxx, "-std=c++17", "-O2", "-Wall", os.path.join(HERE, "cpp", "state_plan_check.cpp"), "-o", exe], check=True)
    r = subprocess.run([exe], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout
