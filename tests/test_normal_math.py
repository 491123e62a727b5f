"""Accuracy of the packed single-precision Box-Muller (rocrand_b200/csrc/normal_math.cuh),
compiled for the host, against double precision: random uniforms and angles, uniforms near 1
and near 0, the floats at and beside the multiples of pi / 2.

Bounds: the logarithm adds one rounding (0.5 ulp) to a sum whose larger term carries at most
half an ulp and a 2^-28 polynomial; a product has three factors' errors -- half the
logarithm's through the square root and its rounding, 1.5 ulp of sine or cosine (two roundings
of the reduced angle's order and the polynomial's), and its own rounding: 4 ulp at most, the
tolerance of the parity tests."""

import os
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(HERE)


def test_box_muller_accuracy(tmp_path):
    nvcc = shutil.which("nvcc")
    if shutil.which("g++") is None or nvcc is None:
        pytest.skip("no host C++ compiler or CUDA headers")
    exe = str(tmp_path / "check")
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-mfma",
                    "-I", os.path.join(ROOT, "rocrand_b200", "csrc"),
                    "-I", os.path.join(os.path.dirname(os.path.dirname(os.path.realpath(nvcc))), "include"),
                    os.path.join(HERE, "normal_math_check.cpp"), "-o", exe], check=True)
    out = subprocess.run([exe, "2000000"], check=True, capture_output=True, text=True).stdout
    rows = {line.split()[0]: [float(v) for v in line.split()[1:]] for line in out.splitlines()}
    assert rows["log"][0] < 1.0, rows
    assert rows["product"][0] < 4.0, rows
    assert rows["norm"][0] < 4.7e-8, rows  # the library form's error on the same kind of inputs
    assert all(v == 0.0 for v in rows["one"]), rows
