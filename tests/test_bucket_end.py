"""GPU: the closing kernel of a bucket batch with inserts, on hand-made state
(compiled here with the kernels' own source)."""
import os
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))


@pytest.mark.gpu
def test_late_device_errors_reach_the_snapshot(lib, tmp_path):
    from ltpmg_gb300 import _build

    exe = str(tmp_path / "end_check")
    _build._run([_build._nvcc()] + _build.ARCH + _build.NVCC_FLAGS +
                [os.path.join(HERE, "buckets", "end_check.cu"), "-o", exe, "-L", _build.PKG, "-lltpmg_gb300",
                 "-Xlinker", "-rpath=" + _build.PKG])
    r = subprocess.run([exe], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0 and r.stdout.strip() == "ok", r.stdout + r.stderr
