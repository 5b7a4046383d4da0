"""Division by a table's spacing (quotientBy, csrc/hs_exact.cuh) against the
plain division on the GPU, bit for bit, on dividends whose quotient lies next to
a double or next to a midpoint between two, where a correction by one last place
decides: the spacings of the workloads' tables, and any divisor."""
import ctypes as C
import os
import subprocess

import pytest

pytestmark = pytest.mark.gpu

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(os.path.dirname(HERE), "moose-core_gb300", "csrc")


@pytest.fixture(scope="module")
def lib():
    out = os.path.join(HERE, "cpp", "_build")
    os.makedirs(out, exist_ok=True)
    so, src = os.path.join(out, "libexact_const_shim.so"), os.path.join(HERE, "cpp", "exact_const_shim.cu")
    nvcc = "/usr/local/cuda/bin/nvcc" if os.path.exists("/usr/local/cuda/bin/nvcc") else "nvcc"
    subprocess.run([nvcc, "-gencode", "arch=compute_103a,code=sm_103a", "-O3", "--fmad=false", "-shared", "-Xcompiler",
                    "-fPIC", "-I", CSRC, "-o", so, src], check=True, capture_output=True, text=True)
    L = C.CDLL(so)
    L.exact_const_check.argtypes = [C.c_double, C.c_ulonglong, C.c_int, C.c_int]
    L.exact_const_check.restype = C.c_longlong
    return L


@pytest.mark.parametrize("d", [0.15 / 3000, 0.15 / 300, 1.0 / 3000, (0.05 - -0.1) / 3000, 1e-3 / 49, 1.0, 0.0])
def test_division_by_a_constant_bit_identical(lib, d):
    assert lib.exact_const_check(d, 77, 304, 1000) == 0        # 8e7 dividends
