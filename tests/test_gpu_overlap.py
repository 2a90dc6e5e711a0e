"""Launches that overlap the kernel before and launches that do not: the same
results on both sides of the sizes where the rule changes."""
import numpy as np
import pytest

from rocflu_gb300 import cases, gpu

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision,sides", [("mixed", (16, 17, 32, 33)), ("fp64", (15, 16, 21, 22)), ("fp64_exact", (15, 16))])
@pytest.mark.parametrize("reconst", [cases.RECONST_BJ, cases.RECONST_WENO_XYZ])
def test_captured_and_host_launched_stages(gpu_lib, precision, sides, reconst):
    """Three steps replayed from the graph and three launched stage by stage:
    equal bits, and equal to the same steps of a second context."""
    for n in sides:
        num = cases.Numerics(space_order=2, space_discr=cases.DISCR_HLLC, reconst=reconst, cfl=0.4)
        c = cases.shock_sphere(n, num=num)
        dt = 0.05 / n
        grid = gpu.Setup(c)
        a, b = gpu.Region(c, precision, grid=grid), gpu.Region(c, precision, grid=grid)
        a.run_fixed_dt(3, dt)
        for _ in range(3):
            b.runge_kutta(dt)
        x, y = a.download()[0], b.download()[0]
        assert np.isfinite(x).all()
        np.testing.assert_array_equal(x, y)
        b.upload(c.cv0)
        for _ in range(3):
            for s in (1, 2, 3):
                gpu.CellGradientsMP(b)
                gpu.ConvectiveFluxesMP(b)
                b.rk_update(s, dt)
        np.testing.assert_array_equal(x, b.download()[0])
