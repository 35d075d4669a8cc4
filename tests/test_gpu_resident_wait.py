"""The resident kernel's bounded wait and its error path: one tile sends no edges
(tests/resident_wait_check.cu), every launch ends by itself, every call reports
the error, and the next run gives the same bits as the one before."""
import os
import subprocess

import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_a_silent_tile_ends_the_launch_with_an_error(tmp_path):
    from fwi_gb300 import build as B
    B.build()
    exe = str(tmp_path / "resident_wait_check")
    short = str(tmp_path / "fwi_resident.o")
    host = str(tmp_path / "resident_wait_check.o")
    cc = [B.nvcc()] + B._flags()
    jobs = [subprocess.Popen(cc + ["-DFWI_RESIDENT_POLLS=5000", "-c", os.path.join(B.CSRC, "fwi_resident.cu"), "-o", short]),
            subprocess.Popen(cc + ["-c", os.path.join(ROOT, "tests", "resident_wait_check.cu"), "-o", host])]
    assert [j.wait() for j in jobs] == [0, 0]
    objs = [os.path.join(B.OUT_DIR, os.path.splitext(f)[0] + ".o") for f in B.SOURCES
            if f not in ("fwi_host.cu", "fwi_resident.cu")]
    subprocess.run([B.nvcc()] + B.ARCH + [host, short] + objs + ["-o", exe, "-cudart", "static", "-lcufft", "-Xlinker",
                                                                "-rpath," + B.CUDA_LIB], check=True)
    r = subprocess.run([exe], capture_output=True, text=True, timeout=120, env=dict(os.environ, FWI_TUNE_CACHE=""))
    assert r.returncode == 0, r.stdout + r.stderr
    assert "wait ok" in r.stdout
