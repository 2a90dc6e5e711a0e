"""The context's device memory (rocflu_gb300/csrc/devmem.h): an array it needs
takes the optional ones' place, whichever came first."""
import os
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))


@pytest.fixture(scope="module")
def prog(tmp_path_factory):
    out = str(tmp_path_factory.mktemp("devmem") / "check")
    subprocess.run(["g++", "-std=c++17", "-O1", "-o", out, os.path.join(HERE, "devmem_check.cpp")], check=True)
    return out


@pytest.mark.parametrize("calls,rows,held", [
    # room for all
    ("need 40 want 30 need 20", ["1 0 0", "1 1 0", "1 1 0"], 90),
    # an optional array that does not fit is left out, the needed ones stay
    ("need 60 want 50 need 30", ["1 0 0", "0 0 0", "1 0 0"], 90),
    # a needed array after them takes their place, once
    ("need 40 want 30 want 20 need 50 need 10", ["1 0 0", "1 1 0", "1 2 0", "1 0 1", "1 0 1"], 100),
    # so does memory that the caller frees itself
    ("need 40 want 50 scratch 60", ["1 0 0", "1 1 0", "1 0 1"], 40),
    # beyond the device: refused, and the optional arrays are gone for good
    ("need 40 want 50 need 70 want 50", ["1 0 0", "1 1 0", "0 0 1", "1 1 1"], 90),
    ("need 40 need 70", ["1 0 0", "0 0 0"], 40),
])
def test_needed_before_optional(prog, calls, rows, held):
    c = calls.split()
    text = "\n".join(" ".join(c[k:k + 2]) for k in range(0, len(c), 2)) + "\n"
    out = subprocess.run([prog, "100"], input=text, capture_output=True, text=True, check=True).stdout.split("\n")
    assert out[:len(rows)] == rows
    assert int(out[len(rows)]) == held and int(out[len(rows) + 1]) == 0
