"""FP64 division, square root and comparisons in integers
(rocflu_gb300/csrc/intmath.h, host code shared with the device) against the C
library's, bit by bit; the device's are counted by rflu_gpu_check_conversions."""
import os
import subprocess

HERE = os.path.dirname(os.path.abspath(__file__))


def test_integer_division_and_root_are_ieee(tmp_path):
    out = str(tmp_path / "check")
    subprocess.run(["g++", "-std=c++17", "-O2", "-o", out, os.path.join(HERE, "intmath_check.cpp")], check=True)
    res = subprocess.run([out, "2000000"], capture_output=True, text=True, check=True)
    assert res.stdout.split()[-1] == "0", res.stdout
