"""The node update's short forms against the general form on the GPU's own
arithmetic, bit for bit (update_device_check.cu)."""
import os
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))


@pytest.mark.gpu
def test_short_forms_bitwise(tmp_path):
    from fm3dt import build
    exe = tmp_path / "check"
    subprocess.run([build.nvcc(), *build.ARCH, "-O3", "-std=c++17", "-fmad=false",
                    os.path.join(HERE, "update_device_check.cu"), "-o", str(exe)],
                   check=True, capture_output=True, text=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stdout + r.stderr
