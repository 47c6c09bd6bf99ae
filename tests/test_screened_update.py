"""The double-precision node update screened in single precision against every
octant solved in double precision, bit for bit, on the host
(screened_update_check.cpp)."""
import os
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))


@pytest.mark.parametrize("seed", [1, 2, 3])
def test_screened_update_bitwise(tmp_path, seed):
    gxx = shutil.which("g++")
    if gxx is None:
        pytest.skip("g++ not found")
    exe = tmp_path / "check"
    subprocess.run([gxx, "-O2", "-std=c++17", "-ffp-contract=off", os.path.join(HERE, "screened_update_check.cpp"),
                    "-o", str(exe)], check=True, capture_output=True, text=True)
    r = subprocess.run([str(exe), "400000", str(seed)], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout + r.stderr
