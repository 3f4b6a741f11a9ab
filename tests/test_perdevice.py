"""Kernel attributes are set on every device that launches
(lace_gb300/csrc/perdevice.h): tests/perdevice_check.cpp compiled with the host
compiler against a stand-in for the CUDA runtime's current device; and no
kernel of the library sets them behind a flag of the whole process without
another way for a launch that is refused."""
import os
import re
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(os.path.dirname(HERE), "lace_gb300", "csrc")


@pytest.mark.skipif(shutil.which("g++") is None, reason="no host C++ compiler")
def test_once_per_device(tmp_path):
    (tmp_path / "cuda_runtime.h").write_text(
        "#pragma once\ntypedef int cudaError_t;\nenum { cudaSuccess = 0 };\ncudaError_t cudaGetDevice(int *);\n")
    exe = str(tmp_path / "perdevice_check")
    subprocess.run(["g++", "-O2", "-std=c++17", "-pthread", "-I", str(tmp_path), "-I", CSRC,
                    os.path.join(HERE, "perdevice_check.cpp"), "-o", exe], check=True)
    r = subprocess.run([exe], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0 and r.stdout.strip() == "ok", (r.returncode, r.stdout, r.stderr)


@pytest.mark.parametrize("name", ["sptrsv_grid.cu", "sptrsv_push.cu", "batch_cluster.cu"])
def test_launchers_set_limits_per_device(name):
    with open(os.path.join(CSRC, name)) as f:
        src = f.read()
    assert "cudaFuncSetAttribute" in src and "static PerDevice" in src
    assert not re.search(r"static\s+const\s+bool\s+\w+\s*=\s*cudaFuncSetAttribute", src)
