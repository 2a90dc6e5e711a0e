"""Derivatives of a first-order residual with a cell without pressure."""
import numpy as np
import pytest

from rocflu_gb300 import cases, gpu

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", ["fp64", "fp64_exact"])
@pytest.mark.parametrize("discr", [cases.DISCR_ROE, cases.DISCR_HLLC, cases.DISCR_AUSM])
def test_adjoint_of_a_cell_without_pressure(gpu_lib, precision, discr):
    """Temperature and sound speed of one cell at rest are zero: the root's
    derivative counts as zero, in the tangent (dual numbers) and in the
    adjoint's closed form alike, so <bar, J dot> = <J' bar, dot>; both sides
    are sums of 5 n products of like size, 1e-12 of the sum of magnitudes."""
    num = cases.Numerics(space_order=1, space_discr=discr, reconst=cases.RECONST_NONE, cfl=0.4)
    c = cases.blast_hex(5, num=num)
    for p in c.patches:
        p.order = 1
    rng = np.random.default_rng(1)
    n = c.n_cells
    rho, p, z = 1.0 + 0.2 * rng.random(n), 1.0 + 0.2 * rng.random(n), np.zeros(n)
    p[n // 2] = 0.0
    c.cv0 = cases.conserved(rho, z, z, z, p, num.gamma)
    dot, bar = rng.standard_normal((2,) + c.cv0.shape)
    r = gpu.Region(c, precision)
    j, v = r.jvp(c.cv0, dot), r.vjp(c.cv0, bar)
    assert np.isfinite(j).all() and np.isfinite(v).all()
    assert abs((bar * j).sum() - (v * dot).sum()) <= 1e-12 * (np.abs(bar * j).sum() + np.abs(v * dot).sum())
