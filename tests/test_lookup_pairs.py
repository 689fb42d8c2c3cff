"""The texels that two lanes fetch for each other's 4D lookups (render
queries), by host arithmetic."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.fixture(scope="module")
def binary(tmp_path_factory):
    if shutil.which("g++") is None:
        pytest.skip("g++ not available")
    out = str(tmp_path_factory.mktemp("cxx") / "lookup_pairs_test")
    # -fwrapv: integers wrap as on the device.
    subprocess.run(["g++", "-std=c++17", "-O1", "-fwrapv",
                    os.path.join(ROOT, "tests", "cxx", "lookup_pairs_test.cc"), "-o", out],
                   check=True, capture_output=True, text=True)
    return out


def test_every_texel_is_in_the_lut(binary):
    """Also for a ray that misses the atmosphere, whose radius has no bound."""
    p = subprocess.run([binary, "bounds"], capture_output=True, text=True, timeout=600)
    assert p.returncode == 0, p.stdout + p.stderr


def test_texels_are_those_of_a_lookup_by_itself(binary):
    """Also where nu is outside its range by rounding, so that a node's columns
    are clamped."""
    p = subprocess.run([binary, "texels"], capture_output=True, text=True, timeout=600)
    assert p.returncode == 0, p.stdout + p.stderr
