"""Two passes side by side: the side stream is joined on every way out."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_side_stream_is_joined_after_a_failure(tmp_path):
    if shutil.which("g++") is None:
        pytest.skip("g++ not available")
    out = str(tmp_path / "fork_test")
    subprocess.run(["g++", "-std=c++17", "-O1",
                    os.path.join(ROOT, "tests", "cxx", "fork_test.cc"), "-o", out],
                   check=True, capture_output=True, text=True)
    p = subprocess.run([out], capture_output=True, text=True, timeout=60)
    assert p.returncode == 0, p.stdout + p.stderr
