"""CPU checks of the resident kernel's plan: the host planner
(fwi_gb300/csrc/fwi_resident_plan.cpp, no CUDA dependency) compiled with g++
together with tests/resident_check.cpp and run over random grids and groups of
shots: tiles partition the grid, every cell has one thread, every index a
thread forms lies inside its array, neighbours agree on what they exchange."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_resident_plans(tmp_path):
    gxx = shutil.which("g++")
    if gxx is None:
        pytest.skip("g++ not available")
    exe = str(tmp_path / "resident_check")
    csrc = os.path.join(ROOT, "fwi_gb300", "csrc")
    subprocess.run([gxx, "-std=c++17", "-O2", "-I", csrc, os.path.join(ROOT, "tests", "resident_check.cpp"),
                    os.path.join(csrc, "fwi_resident_plan.cpp"), os.path.join(csrc, "fwi_lists.cpp"), "-o", exe],
                   check=True)
    r = subprocess.run([exe], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout + r.stderr
    assert "plans ok" in r.stdout
