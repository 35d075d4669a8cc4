"""The snapshot store's division of four cells at once (div4_by_const in
fwi_gb300/csrc/fwi_div.cuh) against CUDA's IEEE division, bit for bit, over quads
that mix zeros, denormals, tiny, ordinary, huge and non-finite dividends, with
and without a reciprocal (0: the division itself)."""
import ctypes as C
import os
import shutil
import subprocess

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    out = str(tmp_path_factory.mktemp("div4") / "div4_check.so")
    subprocess.run([nvcc, "-gencode", "arch=compute_103a,code=sm_103a", "-O3", "-std=c++17", "--fmad=false",
                    "-Xcompiler", "-fPIC", "-shared", "-I", os.path.join(ROOT, "fwi_gb300", "csrc"),
                    os.path.join(ROOT, "tests", "div4_check.cu"), "-o", out], check=True)
    lb = C.CDLL(out)
    lb.div4_check.argtypes = [C.c_float, C.c_float, C.c_uint, C.POINTER(C.c_ulonglong)]
    return lb


@pytest.mark.parametrize("reciprocal", [True, False])
@pytest.mark.parametrize("b", [1e-3, 1.5625e-3, 0.00127797, 7e-4, 0.5, 1.0])
def test_quads_match_ieee_division(lib, b, reciprocal):
    b = np.float32(b)
    y = np.float32(1.0) / b if reciprocal else np.float32(0.0)
    bad = C.c_ulonglong(0)
    assert lib.div4_check(C.c_float(b), C.c_float(y), 1 << 24, C.byref(bad)) == 0
    assert bad.value == 0
