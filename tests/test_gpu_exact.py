"""The FP64 operations of csrc/hs_exact.cuh (division, division by a
constant, compares, integer and fraction part) against the plain operations
on the GPU, bit for bit, on operands where they can go wrong: any bits (NaN,
infinities, zeros, subnormals), short and all-ones mantissas, quotients next
to a power of two and next to a midpoint between two doubles."""
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
    so, src = os.path.join(out, "libexact_shim.so"), os.path.join(HERE, "cpp", "exact_shim.cu")
    nvcc = "/usr/local/cuda/bin/nvcc" if os.path.exists("/usr/local/cuda/bin/nvcc") else "nvcc"
    subprocess.run([nvcc, "-gencode", "arch=compute_103a,code=sm_103a", "-O3", "--fmad=false", "-shared", "-Xcompiler",
                    "-fPIC", "-I", CSRC, "-o", so, src], check=True, capture_output=True, text=True)
    L = C.CDLL(so)
    L.exact_check.argtypes = [C.c_int, C.c_ulonglong, C.c_int, C.c_int]
    L.exact_check.restype = C.c_longlong
    return L


@pytest.mark.parametrize("kind", [0, 1, 2, 3, 4])
def test_operations_bit_identical(lib, kind):
    assert lib.exact_check(kind, 1000 + kind, 608, 2000) == 0      # 3e8 operand pairs
