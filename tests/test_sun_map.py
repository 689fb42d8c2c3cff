"""The mu_s mapping of multiple scattering's ray samples against FP64, by host
arithmetic."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_coordinate_vs_fp64(tmp_path):
    """Maximum sun zenith angles of 10 to 180 degrees."""
    if shutil.which("g++") is None:
        pytest.skip("g++ not available")
    out = str(tmp_path / "sun_map_test")
    subprocess.run(["g++", "-std=c++17", "-O1",
                    os.path.join(ROOT, "tests", "cxx", "sun_map_test.cc"), "-o", out],
                   check=True, capture_output=True, text=True)
    p = subprocess.run([out], capture_output=True, text=True, timeout=600)
    assert p.returncode == 0, p.stdout + p.stderr
