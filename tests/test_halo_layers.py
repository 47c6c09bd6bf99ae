"""The main sweep's halo copies and polls stay inside the event's field when a
wait for the blocks upstream gives up, on the host (halo_layers_check.cpp)."""
import os
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))


def test_halo_layers_stay_in_the_field(tmp_path):
    gxx = shutil.which("g++")
    if gxx is None:
        pytest.skip("g++ not found")
    exe = tmp_path / "check"
    subprocess.run([gxx, "-O2", "-std=c++17", os.path.join(HERE, "halo_layers_check.cpp"), "-o", str(exe)],
                   check=True, capture_output=True, text=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout + r.stderr
