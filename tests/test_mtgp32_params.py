"""The MTGP32 fill reads up to pos + 255 words ahead in a ring with 96 words repeated behind it: the
embedded parameter sets keep to that, and others are refused before any kernel sees them."""

import os
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(HERE)


def test_pos_in_range(tmp_path):
    if shutil.which("g++") is None:
        pytest.skip("no host C++ compiler")
    exe = str(tmp_path / "check")
    subprocess.run(["g++", "-O2", "-std=c++17", "-I", os.path.join(ROOT, "rocrand_b200", "csrc"),
                    os.path.join(HERE, "mtgp32_params_check.cpp"), "-o", exe], check=True)
    blob = os.path.join(ROOT, "rocrand_b200", "data", "mtgp32_params.bin")
    low, high, *refused = subprocess.run([exe, blob], check=True, capture_output=True, text=True).stdout.split()
    assert 1 <= int(low) <= int(high) <= 95
    assert refused == ["1"] * 7
