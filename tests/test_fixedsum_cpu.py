"""The fixed-point sums of products (rocflu_gb300/csrc/fixedsum.h, host code
shared with the device) against exact rational sums."""
import math
import os
import subprocess
from fractions import Fraction

import numpy as np
import pytest

HERE = os.path.dirname(os.path.abspath(__file__))


@pytest.fixture(scope="module")
def prog(tmp_path_factory):
    out = str(tmp_path_factory.mktemp("fixedsum") / "check")
    subprocess.run(["g++", "-std=c++17", "-O2", "-o", out, os.path.join(HERE, "fixedsum_check.cpp")], check=True)
    return out


def _run(prog, cases):
    lines = []
    for own, q, w in cases:
        lines.append(" ".join([str(len(q)), float(own).hex()] + [float(x).hex() for p in zip(q, w) for x in p]))
    res = subprocess.run([prog], input="\n".join(lines) + "\n", capture_output=True, text=True, check=True)
    return res.stdout.split()


def _bound(own, q, w):
    """Every value is cut to a unit of 2^-55 of the power of two above the
    largest, every weight rounded to one of the largest weight's, the result
    to a double."""
    def unit(v):
        top = max(abs(float(x)) for x in v)
        return Fraction(2) ** (math.frexp(top)[1] - 55) if top else Fraction(0)

    uq, uw = unit(list(q) + [own]), unit(w)
    diff = [Fraction(x) - Fraction(own) for x in q]
    exact = sum((Fraction(a) * d for a, d in zip(w, diff)), Fraction(0))
    err = uq * sum(abs(Fraction(a)) for a in w) + uw / 2 * sum(abs(d) + uq for d in diff)
    return exact, err + abs(exact) * Fraction(2) ** -53


@pytest.mark.parametrize("kind", ["near", "signed", "ratio", "tiny", "huge", "ties"])
def test_sums_within_their_units(prog, kind):
    rng = np.random.default_rng(4)
    cases = []
    for t in range(400):
        n = int(rng.choice([1, 2, 7, 26, 40, 64]))
        u = rng.uniform(-1, 1, n + 1)
        q = {"near": 3.7 * (1 + 2.0 ** -int(rng.integers(0, 52)) * u), "signed": u * 2.0 ** rng.integers(-9, 9),
             "ratio": u * 2.0 ** rng.integers(-60, 1, n + 1), "tiny": u * 2.0 ** -480, "huge": u * 2.0 ** 480,
             "ties": np.where(u > 0, 1.0, -1.0)}[kind]
        w = rng.uniform(-1, 1, n) * 2.0 ** rng.integers(-8, 20)
        if kind == "ties":  # the largest partial products all of one sign
            w = np.where(q[1:] > 0, 1.0, -1.0) * (2.0 - 2.0 ** -52)
            q[0] = -1.0
        cases.append((q[0], q[1:], w))
    for (own, q, w), got in zip(cases, _run(prog, cases)):
        exact, err = _bound(own, q, w)
        assert abs(Fraction(float.fromhex(got)) - exact) <= err


def test_zeros_and_what_is_left_to_fp64(prog):
    z = [0.0, -0.0]
    got = _run(prog, [(0.0, z, [1.0, 2.0]), (-0.0, [1.0, 1.0], [1.0, -1.0]), (2.0, [2.0, 2.0], [0.3, 7.0]),
                      (math.inf, [1.0], [1.0]), (1.0, [math.nan], [1.0]), (1.0, [5e-310], [1.0]),
                      (1.0, [1e200], [1.0]), (1.0, [2.0], [0.0]), (1.0, [2.0] * 65, [1.0] * 65)])
    assert [float.fromhex(g) for g in got[:3]] == [0.0, 0.0, 0.0]
    assert got[3:] == ["bad"] * 6
