"""The library's host code on a stand-in for the GPU (tests/cpp/fake_cuda.cpp),
compiled here with g++: ``load()`` as a context in which the package's classes
run on it.  Kernels do nothing but reinit; what is tested is the host path."""
import contextlib
import ctypes as C
import os
import shutil
import subprocess

from moose_gb300 import _native

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(os.path.dirname(HERE), "moose-core_gb300", "csrc")
OUT = os.path.join(HERE, "cpp", "_build")


def _build():
    os.makedirs(OUT, exist_ok=True)
    so = os.path.join(OUT, "libfake_gpu.so")
    units = [os.path.join(CSRC, u) for u in ("hs_api.cpp", "hs_batch_api.cpp", "hs_plan.cpp", "hs_cell.cu")]
    units.append(os.path.join(HERE, "cpp", "fake_cuda.cpp"))
    deps = units + [os.path.join(CSRC, f) for f in os.listdir(CSRC)]
    if os.path.exists(so) and os.path.getmtime(so) >= max(map(os.path.getmtime, deps)):
        return so
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    inc = os.path.join(os.path.dirname(os.path.dirname(os.path.realpath(nvcc))), "include")
    flags = ["-O2", "-std=c++17", "-fPIC", "-ffp-contract=off", "-fvisibility=default", "-I", CSRC, "-I", inc]
    objs = [os.path.join(OUT, os.path.basename(u) + ".fake.o") for u in units]
    procs = [subprocess.Popen(["g++"] + flags + ["-x", "c++", "-c", u, "-o", o], stderr=subprocess.PIPE, text=True)
             for u, o in zip(units, objs)]
    for p in procs:
        err = p.communicate()[1]
        assert p.returncode == 0, err
    subprocess.run(["g++", "-shared", "-Wl,-Bsymbolic", "-o", so] + objs + ["-lpthread"], check=True,
                   capture_output=True, text=True)
    return so


@contextlib.contextmanager
def load():
    so = _build()
    kept, path = _native._LIB, _native.lib_path
    _native._LIB, _native.lib_path = None, lambda: so
    try:
        L = _native.load()
        L.fake_lazy.argtypes = [C.c_int, C.c_int]
        L.fake_table.argtypes = [C.c_uint32, C.POINTER(C.c_uint32)]
        L.fake_table.restype = C.POINTER(C.c_double)
        L.fake_allow.argtypes = L.fake_limit.argtypes = [C.c_uint64, C.c_int]
        L.fake_digest.argtypes, L.fake_digest.restype = [C.c_uint64], C.c_uint64
        L.fake_cell_bytes.restype = C.c_uint64
        yield L
        L.fake_lazy(0, 0)
    finally:
        _native._LIB, _native.lib_path = kept, path
