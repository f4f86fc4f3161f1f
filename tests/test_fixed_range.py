"""The fixed-point functions of FP64 stepping have no undefined arithmetic,
whatever the position, and refuse positions outside their range."""
import os
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))


@pytest.mark.parametrize("flags", [["-fsanitize=undefined", "-fsanitize-undefined-trap-on-error"], ["-ftrapv"]])
def test_no_undefined_arithmetic(tmp_path, flags):
    exe = str(tmp_path / "fixed_range")
    subprocess.run(["g++", "-O1", "-std=c++17", *flags, os.path.join(HERE, "cpp", "fixed_range_main.cpp"), "-o", exe], check=True)
    out = subprocess.run([exe], capture_output=True, text=True)
    assert out.returncode == 0 and out.stdout.startswith("ok"), (out.returncode, out.stdout)
