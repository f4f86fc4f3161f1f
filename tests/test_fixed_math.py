"""The fixed-point functions of FP64 stepping (fk_fixed.cuh), compiled for the
host and compared with long double: each within the error bound that its
number format gives, and none less exact than the FP64 form it replaces."""
import os
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))


@pytest.fixture(scope="module")
def errors(tmp_path_factory):
    exe = str(tmp_path_factory.mktemp("fx") / "fixed_math")
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", os.path.join(HERE, "cpp", "fixed_math_main.cpp"), "-o", exe],
                   check=True)
    out = subprocess.run([exe], check=True, capture_output=True, text=True).stdout
    return {w[0]: [float(v) for v in w[1:]] for w in (line.split() for line in out.splitlines())}


@pytest.mark.parametrize("name,bound", [
    ("exp_ulp", 1.3),             # units of 2^-53: the result's rounding 1, the exponent's 2^-55 1/4, products 2^-58
    ("neg_log_abs", 2.0 ** -55),  # 16 units of 2^-59
    ("sincos_abs", 2.0 ** -58),   # theta^5 / 120 at theta = pi / 4096, and products low by 2 units of 2^-63
    ("sqrt_ulp", 2.0 ** -4),      # units of 2^-53: 2^-57
    ("normal_fx_abs", 2.0 ** -53),  # rounding to 2^-53 units, and the pair's own 2^-54 at |z| up to 6.8
])
def test_bounds(errors, name, bound):
    assert errors[name][0] <= bound


def test_normal_pair_no_less_exact_than_fp64(errors):
    assert errors["normal_abs"][0] <= errors["normal_abs_fp64"][0]
    assert errors["normal_rms"][0] <= errors["normal_rms_fp64"][0]


@pytest.mark.parametrize("name", ["lap", "u", "ux", "uy", "lap_terms", "a", "sigma", "f", "mc", "Ux", "Uy"])
def test_problem_functions_no_less_exact_than_fp64(errors, name):
    for key in (name, name + "_max"):
        fixed, fp64 = errors[key]
        assert fixed <= fp64, key
