"""Shared-memory limits are raised per device (ltpmg_gb300/csrc/ltp_smem.h;
CPU, compiled here against stand-ins for the runtime calls), and by every
kernel launch that needs more than the default."""
import glob
import os
import re
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(os.path.dirname(HERE), "ltpmg_gb300", "csrc")


def test_limit_is_raised_once_per_device(tmp_path):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(nvcc):
        pytest.skip("no CUDA headers")
    inc = os.path.join(os.path.dirname(os.path.dirname(os.path.realpath(nvcc))), "include")
    exe = str(tmp_path / "smem_check")
    subprocess.run(["g++", "-std=c++17", "-O1", "-I", inc, os.path.join(HERE, "smem", "smem_check.cpp"), "-o", exe,
                    "-lpthread"], check=True)
    r = subprocess.run([exe], capture_output=True, text=True)
    assert r.returncode == 0 and r.stdout.strip() == "ok", r.stdout + r.stderr


def test_no_limit_is_raised_another_way():
    for path in glob.glob(os.path.join(CSRC, "*.cu*")) + glob.glob(os.path.join(CSRC, "*.cpp")):
        with open(path) as f:
            assert not re.search(r"cudaFuncSetAttribute", f.read()), path
