"""MRG32k3a's folded remainders against %, over edge states (tests/mrg_step_check.cpp)."""

import os
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(HERE)


def test_step_equals_plain_remainders(tmp_path):
    if shutil.which("nvcc") is None:
        pytest.skip("no nvcc")
    exe = str(tmp_path / "check")
    subprocess.run(["nvcc", "-O2", "-std=c++17", "-gencode", "arch=compute_100a,code=sm_100a", "-x", "cu",
                    "-I", os.path.join(ROOT, "rocrand_b200", "csrc"), "-I", os.path.join(ROOT, "include"),
                    os.path.join(HERE, "mrg_step_check.cpp"), "-o", exe], check=True)
    bad, count = subprocess.run([exe], check=True, capture_output=True, text=True).stdout.split()
    assert int(count) > 3000000 and int(bad) == 0
