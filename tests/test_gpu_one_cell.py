"""A mesh of one cell: no interior face, no stencil."""
from types import SimpleNamespace

import numpy as np
import pytest

from rocflu_gb300 import cases, gpu

pytestmark = pytest.mark.gpu


def _unit_cube():
    n = np.array([[-1, 0, 0], [1, 0, 0], [0, -1, 0], [0, 1, 0], [0, 0, -1], [0, 0, 1]], float)
    return SimpleNamespace(f2c=np.zeros((0, 2), np.int32), fn=np.zeros((0, 4)), fc=np.zeros((0, 3)), vol=np.ones(1),
                           cofg=np.full((1, 3), 0.5), patch_off=np.arange(7, dtype=np.int32),
                           bf2c=np.ones(6, np.int32), bfn=np.column_stack([n, np.ones(6)]), bfc=0.5 + 0.5 * n,
                           c2cs_off=np.zeros(2, np.int32), c2cs=np.zeros(0, np.int32), moms=np.zeros((1, 10)))


@pytest.mark.parametrize("precision", ["fp64", "fp64_exact"])
def test_read_out_of_one_cell(gpu_lib, precision):
    """Gradients and residual of one cell at rest between walls: no gradient,
    the pressure's forces cancel.  (One cell's gradient array has the packed
    records' unit stride.)"""
    c = cases.shock_sphere(1, num=cases.Numerics(space_order=2, reconst=cases.RECONST_NONE))
    for p in c.patches:
        p.bc_type, p.order = cases.BC_SLIPWALL, 1
    z = np.zeros(1)
    c.cv0 = cases.conserved(np.full(1, 1.3), z, z, z, np.full(1, 0.7), c.num.gamma)
    r = gpu.Region(c, precision, grid=_unit_cube())
    rhs, grad = r.residual(c.cv0)
    np.testing.assert_array_equal(grad, np.zeros((1, 5, 3)))
    np.testing.assert_array_equal(rhs, np.zeros((1, 5)))
    gpu.CellGradientsMP(r)
    np.testing.assert_array_equal(r.get_grad(), np.zeros((1, 5, 3)))
