"""GPU: how a bucket batch ends when a device error was noted: the closing
kernel of a batch with inserts, and the error exit of the skew fallback, on
hand-made state (compiled here)."""
import os
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))


@pytest.mark.gpu
@pytest.mark.parametrize("name", ["end_check", "fallback_check"])
def test_device_errors_end_a_batch_in_order(lib, tmp_path, name):
    from ltpmg_gb300 import _build

    exe = str(tmp_path / name)
    _build._run([_build._nvcc()] + _build.ARCH + _build.NVCC_FLAGS +
                [os.path.join(HERE, "buckets", name + ".cu"), "-o", exe, "-L", _build.PKG, "-lltpmg_gb300",
                 "-Xlinker", "-rpath=" + _build.PKG])
    r = subprocess.run([exe], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0 and r.stdout.strip() == "ok", r.stdout + r.stderr
