"""CPU check of the resident kernel's number of shots per launch: the host
planner compiled with g++ together with tests/resident_group_check.cpp, its
reported time against the plain sum over the launches."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_group_time_is_the_sum_of_its_launches(tmp_path):
    gxx = shutil.which("g++")
    if gxx is None:
        pytest.skip("g++ not available")
    exe = str(tmp_path / "resident_group_check")
    csrc = os.path.join(ROOT, "fwi_gb300", "csrc")
    subprocess.run([gxx, "-std=c++17", "-O2", "-I", csrc, os.path.join(ROOT, "tests", "resident_group_check.cpp"),
                    os.path.join(csrc, "fwi_resident_plan.cpp"), os.path.join(csrc, "fwi_lists.cpp"), "-o", exe],
                   check=True)
    r = subprocess.run([exe], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout + r.stderr
    assert "groups ok" in r.stdout
