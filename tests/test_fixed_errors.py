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
    lines = _lines(tmp_path_factory, "fixed_normals")
    assert {int(w[0]) for w in lines} >= set(range(-16, 3))  # radius 2^-16 (u next to 1) to 6.8
    for w in lines:
        rms, top, rms64, top64 = map(float, w[1:])
        assert rms <= rms64 and top <= top64, w
