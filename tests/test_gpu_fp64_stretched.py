"""The FP64 mode's gradients on stretched and graded meshes."""
import numpy as np
import pytest

from rocflu_gb300 import cases, gpu
from test_fixedsum_cells_cpu import in_fixed_point, stencil_weights, stretched

pytestmark = pytest.mark.gpu


def _graded():
    """Cubic cells with one layer of 40:1 cells on the high x side: cells in
    fixed point beside cells in FP64, also within a warp."""
    c = cases.shock_sphere(16, num=cases.Numerics(space_order=2, reconst=cases.RECONST_NONE))
    x = c.xyz[:, 0]
    c.xyz[:, 0] = np.where(x > 1 - 1 / 32, x + 39 / 16, x)
    c.xyz = np.ascontiguousarray(c.xyz)
    return c, gpu.Setup(c)


def _gradient_errors(region, cv, s, ext):
    """Per cell, variable and component: the gradient's error against sums in
    extended precision over the same primitive state, sum |w||d| of the
    component and, with the member's largest weight, of the cell."""
    _, g = region.residual(cv)
    region.upload(cv)
    _, dv = region.download()
    ir = 1.0 / cv[:, 0]
    q = np.column_stack([cv[:, 0], ir * cv[:, 1], ir * cv[:, 2], ir * cv[:, 3], dv[:, 0]]).astype(np.longdouble)
    row, idx, w = stencil_weights(s)
    off = s.c2cs_off[:-1]
    d = q[idx] - q[row]
    exact = np.stack([np.add.reduceat(w[:, c:c + 1].astype(np.longdouble) * d, off) for c in range(3)], axis=2)
    size = np.stack([np.add.reduceat(np.abs(w[:, c:c + 1] * d), off) for c in range(3)], axis=2).astype(float)
    whole = np.add.reduceat(np.abs(w).max(axis=1)[:, None] * np.abs(d), off).astype(float)
    return np.abs(g - exact).astype(float), size, whole


@pytest.mark.parametrize("mesh,aspect", [("hex", 1), ("tets", 1), ("hex", 2), ("tets", 2), ("hex", 100), ("tets", 100),
                                         ("hex", 1e4), ("tets", 1e4), ("graded", 1)])
def test_gradients_on_stretched_cells(gpu_lib, mesh, aspect):
    """Against sums in extended precision: the cells in fixed point are rounded
    no more than the FP64_EXACT mode's, as vectors and in the root mean square;
    each component of those in FP64 is within the bound of an FP64 sum of n
    products, (n + 3) 2^-53 of sum |w d| (n products and sums, and the
    difference)."""
    c, s = _graded() if mesh == "graded" else stretched(mesh, aspect)
    rng = np.random.default_rng(6)
    n, ext = s.n_cells, s.cofg.max(axis=0)
    y = s.cofg / ext
    wave = [np.sin(y @ rng.uniform(1, 4, 3) + rng.uniform(0, 6)) for _ in range(5)]
    u = [0.3 * wave[k] + 0.2 * s.cofg[:, 0] + 0.02 * rng.standard_normal(n) for k in range(3)]
    rho, p = 1.0 + 0.3 * wave[3], np.where(y @ [1.0, 0.7, 0.4] < 1.0, 100.0, 1.0) * (1.0 + 0.2 * wave[4])
    p = p + 0.5 * rho * max(float((a * a).max()) for a in u)  # clear of the energy's rounding
    cv = cases.conserved(rho, *u, p, c.num.gamma)
    c.cv0 = cv
    members = np.diff(s.c2cs_off)[:, None, None]
    err, size, whole = _gradient_errors(gpu.Region(c, "fp64", grid=s), cv, s, ext)
    ref, _, _ = _gradient_errors(gpu.Region(c, "fp64_exact", grid=s), cv, s, ext)
    fixed = in_fixed_point(s, stencil_weights(s)[2])
    assert fixed.any() == (aspect <= 2) and fixed.all() == (aspect == 1 and mesh != "graded")
    if fixed.any():
        a, b = err[fixed].max(axis=2) / whole[fixed], ref[fixed].max(axis=2) / whole[fixed]
        assert (np.sqrt((a * a).mean(axis=0)) <= np.sqrt((b * b).mean(axis=0))).all(), (mesh, aspect)
    bound = (members + 3) * 2.0 ** -53 * size + 1e-300
    assert (err <= bound)[~fixed].all(), float((err / bound)[~fixed].max())
