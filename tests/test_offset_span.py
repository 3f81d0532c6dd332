"""Offsets beyond 32 bits inside one block: the plans tell the kernels not to
tabulate them (host rule; no block of that size is allocated)."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_mappings_beyond_32_bits_are_found(tmp_path):
    if not shutil.which("g++"):
        pytest.skip("g++ not available")
    exe = str(tmp_path / "offset_span_test")
    r = subprocess.run(["g++", "-std=c++17", "-O1", "-Wall", "-Werror", "-I", os.path.join(ROOT, "libtensor_b200", "csrc"),
                        os.path.join(ROOT, "tests", "cpp", "offset_span_test.cpp"), "-o", exe],
                       capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    r = subprocess.run([exe], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0, r.stdout
