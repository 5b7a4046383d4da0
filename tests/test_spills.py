"""Registers of the mixed stepping kernels: 1,024 threads have 64 each, and a
spilled one costs an L2 access where shared memory leaves little L1.  Every
instantiation keeps what it needs in them but for a few bytes, as nvcc
reports it."""
import os
import re
import shutil
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "moose-core_gb300", "csrc")
FEW = 16            # bytes: two registers stored, or four read back


def test_stepping_kernels_do_not_spill(tmp_path):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(nvcc):
        pytest.skip("no nvcc")
    r = subprocess.run([nvcc, "-gencode", "arch=compute_103a,code=sm_103a", "-lineinfo", "-O3", "-std=c++17", "-Xptxas",
                        "-v", "-c", os.path.join(CSRC, "hs_mixed.cu"), "-o", str(tmp_path / "o.o")],
                       capture_output=True, text=True)
    assert r.returncode == 0, r.stderr[-2000:]
    seen, over, name = 0, {}, ""
    for line in r.stderr.splitlines():
        m = re.search(r"entry function '(\w+)'", line)
        name = m.group(1) if m else name
        m = re.search(r"(\d+) bytes spill stores, (\d+) bytes spill loads", line)
        if m and "hsForest" in name:
            seen += 1
            if max(map(int, m.groups())) > FEW:
                over[name] = m.groups()
    assert seen >= 10
    assert not over
