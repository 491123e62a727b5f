"""Edges of the fp64 sine / cosine table and of the uniform's logarithm (precise_math.cuh)."""

import os
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(HERE)


def test_edges(tmp_path):
    if shutil.which("g++") is None:
        pytest.skip("no host C++ compiler")
    csrc = os.path.join(ROOT, "rocrand_b200", "csrc")
    subprocess.run(["make", "-s", "-C", csrc, "../../_build/data/precise_tables.inc"], check=True,
                   capture_output=True)
    exe = str(tmp_path / "check")
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-I", csrc,
                    "-I", os.path.join(ROOT, "_build", "data"), os.path.join(HERE, "precise_circle_check.cpp"),
                    "-o", exe, "-lquadmath"], check=True)
    worst, miss, count, differ = subprocess.run([exe], check=True, capture_output=True,
                                                text=True).stdout.split()
    # half an ulp, plus 2^-10 for the internal error (test_precise_math.py's bound)
    assert float(worst) <= 0.5 + 2.0 ** -10, worst
    assert int(miss) <= 1e-4 * int(count), (miss, count)
    assert int(differ) == 0
