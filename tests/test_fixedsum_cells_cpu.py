"""The fixed-point sums of whole cells (rocflu_gb300/csrc/fixedsum.h) on the
stencils of stretched meshes, against exact rational sums: which cells the
fixed point takes, and that it is no less accurate there than FP64 sums."""
import os
import subprocess
from fractions import Fraction

import numpy as np
import pytest

from rocflu_gb300 import cases, gpu

HERE = os.path.dirname(os.path.abspath(__file__))


@pytest.fixture(scope="module")
def prog(tmp_path_factory):
    out = str(tmp_path_factory.mktemp("fixedcells") / "check")
    subprocess.run(["g++", "-std=c++17", "-O2", "-ffp-contract=off", "-o", out,
                    os.path.join(HERE, "fixedsum_cells_check.cpp")], check=True)
    return out


def stencil_weights(s):
    """(row, member, weight (nnz, 3)): the least-squares weights as the context forms them from the set-up's moments."""
    row = np.repeat(np.arange(s.n_cells), np.diff(s.c2cs_off))
    idx = s.c2cs - 1
    r11, r12, r22, r13, r23, r33 = (s.moms[:, k] for k in range(6))
    c11, c22, c33 = 1 / r11, 1 / r22, 1 / r33
    c12 = -c11 * r12
    c13, c23 = -(c11 * r13 + c12 * c22 * r23), -c22 * r23
    d = s.cofg[idx] - s.cofg[row]
    t = 1 / np.sqrt(d[:, 0] * d[:, 0] + d[:, 1] * d[:, 1] + d[:, 2] * d[:, 2])
    x, y, z = (t * d[:, k] for k in range(3))
    t1, t2 = (c11 * c11)[row] * x, (c22 * c22)[row] * (y + c12[row] * x)
    t3 = (c33 * c33)[row] * (z + c23[row] * y + c13[row] * x)
    return row, idx, np.stack([t * (t1 + c12[row] * t2 + c13[row] * t3), t * (t2 + c23[row] * t3), t * t3], axis=1)


def in_fixed_point(s, w):
    """The cells whose weights are of like size: the exponents of the components' largest within 2 of each other,
    those of the members' largest within 6."""
    e = np.frexp(np.abs(w))[1]
    e = np.where(w == 0, -2000, e)
    off = s.c2cs_off[:-1]
    comp, member = np.maximum.reduceat(e, off), e.max(axis=1)
    return (member.max() < 600) & (np.ptp(comp, axis=1) <= 2) & \
        (np.maximum.reduceat(member, off) - np.minimum.reduceat(member, off) <= 6)


def stretched(mesh, aspect):
    num = cases.Numerics(space_order=2, reconst=cases.RECONST_NONE)
    c = cases.shock_sphere(6, num=num) if mesh == "hex" else cases.adjoint_tets(4, num=num)
    c.xyz = np.ascontiguousarray(c.xyz * np.array([aspect, 1.0, 1.0]))
    return c, gpu.Setup(c)


def _fields(x, aspect):
    rng = np.random.default_rng(3)
    u = rng.uniform(-1, 1, len(x))
    y = x / np.array([aspect, 1.0, 1.0])
    return {"random": u, "linear": 1.3 + 0.37 * x[:, 0] - 0.2 * x[:, 1],
            "smooth": np.sin(3 * y[:, 0]) * np.cos(2 * y[:, 1]) + 0.1 * np.sin(4 * y[:, 2]),
            "jump": np.where(y @ [1.0, 0.7, 0.4] < 1.0, 1e3, 1.0) * (1 + 0.05 * u)}


@pytest.mark.parametrize("mesh", ["hex", "tets"])
@pytest.mark.parametrize("aspect", [1, 2, 16, 1e4])
def test_cells_no_less_accurate_than_fp64(prog, mesh, aspect):
    """Cubic cells all in fixed point, slender ones none; over the cells it
    takes, the root mean square of the gradient's error in units of
    sum |w||d| is at most the FP64 loop's."""
    _, s = stretched(mesh, aspect)
    row, idx, w = stencil_weights(s)
    off, takes = s.c2cs_off, in_fixed_point(s, w)
    for name, q in _fields(s.cofg, aspect).items():
        lines = []
        for i in range(s.n_cells):
            m = range(off[i], off[i + 1])
            lines.append(" ".join([str(len(m)), float(q[i]).hex()] +
                                  [float(v).hex() for k in m for v in (q[idx[k]], *w[k])]))
        got = subprocess.run([prog], input="\n".join(lines) + "\n", capture_output=True, text=True, check=True).stdout
        fixed, loop = [], []
        for i, line in enumerate(got.splitlines()):
            f = line.split()
            assert (f[0] == "fixed") == takes[i]
            if f[0] != "fixed":
                continue
            m = range(off[i], off[i + 1])
            d = [Fraction(float(q[idx[k]])) - Fraction(float(q[i])) for k in m]
            size = float(sum(abs(x) * Fraction(float(np.abs(w[k]).max())) for x, k in zip(d, m)))
            if size == 0.0:
                continue
            exact = [sum(Fraction(float(w[k, c])) * x for x, k in zip(d, m)) for c in range(3)]
            err = [max(abs(float(Fraction(float.fromhex(f[1 + p + c])) - exact[c])) for c in range(3)) / size for p in (0, 3)]
            fixed.append(err[0])
            loop.append(err[1])
        if aspect == 1:
            assert len(fixed) == s.n_cells, name
        if aspect >= 16:
            assert not fixed, name
        if fixed:
            assert np.sqrt(np.mean(np.square(fixed))) <= np.sqrt(np.mean(np.square(loop))), name


def test_weights_out_of_range_stay_in_fp64(prog):
    """Weights so small that a sum would leave the normal doubles."""
    def cell(scale, value):
        w = scale * np.array([[1.0, 0.5, 0.25], [-0.5, 1.0, 0.5], [0.25, -0.5, 1.0]])
        return " ".join(["3", float(value).hex()] + [float(v).hex() for k in range(3) for v in (value * (k + 2), *w[k])])

    out = subprocess.run([prog], input="\n".join([cell(2.0 ** -411, 2.0 ** -499), cell(2.0 ** -430, 2.0 ** -499),
                                                  cell(2.0 ** -411, 1.0)]) + "\n", capture_output=True, text=True,
                         check=True).stdout.splitlines()
    assert [x.split()[0] for x in out] == ["fixed", "fp64", "fixed"]
    for x, v in ((out[0], 2.0 ** -910), (out[2], 2.0 ** -411)):
        f = [float.fromhex(y) for y in x.split()[1:]]
        assert f[:3] == f[3:] == [v * y for y in (0.75, 1.0, 4.25)], f
