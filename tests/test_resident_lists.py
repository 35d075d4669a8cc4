"""CPU check of the resident kernel's launches where sources and receivers fill
the tiles' shared memory: the host planner compiled with g++ together with
tests/resident_lists_check.cpp."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_launches_make_room_for_sources_and_receivers(tmp_path):
    gxx = shutil.which("g++")
    if gxx is None:
        pytest.skip("g++ not available")
    exe = str(tmp_path / "resident_lists_check")
    csrc = os.path.join(ROOT, "fwi_gb300", "csrc")
    subprocess.run([gxx, "-std=c++17", "-O2", "-I", csrc, "-I", os.path.join(ROOT, "tests"),
                    os.path.join(ROOT, "tests", "resident_lists_check.cpp"), os.path.join(csrc, "fwi_resident_plan.cpp"),
                    os.path.join(csrc, "fwi_lists.cpp"), "-o", exe], check=True)
    r = subprocess.run([exe], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout + r.stderr
    assert "lists ok" in r.stdout
