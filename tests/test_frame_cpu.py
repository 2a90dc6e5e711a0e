"""The FP64 mode's eigen-frame (rocflu_gb300/csrc/frame_fp64.cuh, host code
shared with the device): finite and orthonormal for strain rates of any size,
and no further from diagonal than the Jacobi loop it stands for."""
import os
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))


@pytest.fixture(scope="module")
def prog(tmp_path_factory):
    out = str(tmp_path_factory.mktemp("frame") / "check")
    subprocess.run(["g++", "-std=c++17", "-O2", "-w", "-I", os.path.join(HERE, "..", "rocflu_gb300", "csrc"), "-o", out,
                    os.path.join(HERE, "frame_check.cpp")], check=True)
    return out


def _run(prog, mode):
    return subprocess.run([prog, mode], capture_output=True, text=True, check=True).stdout.split("\n")


def test_frames_of_any_size(prog):
    assert _run(prog, "sizes")[0] == "0"


def test_frame_no_less_accurate_than_the_loop(prog):
    """Root mean square and largest remainder over 40,000 matrices a family."""
    for line in _run(prog, "residual")[:2]:
        rms0, rms1, top0, top1, orth0, orth1 = map(float, line.split())
        assert rms1 <= rms0 and top1 <= top0 and orth1 <= orth0, line
