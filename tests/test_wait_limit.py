"""A sweep whose upstream columns never come ends by itself and reports it
(wait_limit_check.cu), in both precisions, all forms."""
import os
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))


@pytest.mark.gpu
def test_waits_give_up(tmp_path):
    from fm3dt import build
    exe = tmp_path / "check"
    subprocess.run([build.nvcc(), *build.ARCH, "-O3", "-std=c++17", "--expt-relaxed-constexpr", "-fmad=false",
                    "-DFM_WAIT_POLLS=4096", os.path.join(HERE, "wait_limit_check.cu"), "-o", str(exe)],
                   check=True, capture_output=True, text=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stdout + r.stderr
