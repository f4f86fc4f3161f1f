"""The fixed-point functions of FP64 stepping (fk_fixed.cuh) beside the FP64
forms that they replace, both against long double: no larger error wherever
in their range, not only in a mean over all of it."""
import os
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))


def _lines(tmp_path_factory, name):
    exe = str(tmp_path_factory.mktemp("fx") / name)
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", os.path.join(HERE, "cpp", name + "_main.cpp"), "-o", exe],
                   check=True)
    out = subprocess.run([exe], check=True, capture_output=True, text=True).stdout
    return [line.split() for line in out.splitlines()]


def test_normal_pair_by_radius(tmp_path_factory):
    fx, *lines = _lines(tmp_path_factory, "fixed_normals")
    assert fx[0] == "fx" and float(fx[1]) <= 0.5  # rounded to nearest
    assert {int(w[0]) for w in lines} >= set(range(-16, 3))  # radius 2^-16 (u next to 1) to 6.8
    for w in lines:
        rms, top, rms64, top64 = map(float, w[1:])
        assert rms <= rms64 and top <= top64, w


def test_problem_functions_by_cell(tmp_path_factory):
    """Every function in every cell of the range.  Where the last rounding to a
    double is all of the error on both sides (a, sigma and -c, of order 1), the
    two rms agree to the noise of 1,500 samples: 1 / sqrt(2 n) = 2 % each."""
    lines = _lines(tmp_path_factory, "fixed_cells")
    assert len(lines) == 14 * 14 * 11
    for w in lines:
        rms, mean, top, rms64, _, top64 = map(float, w[3:])
        slack = 1.02 if w[0] in ("a", "sigma", "mc") else 1.0
        assert rms <= slack * rms64 and top <= slack * top64, w
        # what does not average out over a path's steps
        assert abs(mean) <= 0.5 * rms64, w
