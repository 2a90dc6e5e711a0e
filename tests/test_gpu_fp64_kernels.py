"""FP64 kernels on the device at the sizes where a launch or a kernel branch
changes, against the CPU oracle."""
import numpy as np
import pytest

from oracle.oracle import Oracle
from rocflu_gb300 import cases, gpu

pytestmark = pytest.mark.gpu


def _wavy(case, seed=5, amp=0.01):
    """The case's state with every variable disturbed."""
    rng = np.random.default_rng(seed)
    cv = case.cv0 * (1.0 + amp * rng.standard_normal(case.cv0.shape))
    cv[:, 1:4] += amp * rng.standard_normal((len(cv), 3))
    return cv


@pytest.mark.parametrize("nx", [1, 31, 33, 3041, 4871, 9728, 9729, 19457, 38913])
def test_launch_shapes_bit_exact(gpu_lib, nx):
    """Blocks of 32 to 256 threads and their remainders (4 nx cells): two
    first-order steps, FP64_EXACT, equal to the oracle's bits."""
    c = cases.sod(nx, 2, 2)
    c.cv0 = _wavy(c)
    c.num.dt_imposed = 1e-6
    o = Oracle(c)
    o.set_state(c.cv0)
    n_o, t_o = o.run(2, 1.0)
    r = gpu.Region(c, "fp64_exact")
    n_g, t_g, rc = r.step(2, 1.0)
    assert rc == 0 and n_g == n_o and t_g == t_o
    np.testing.assert_array_equal(r.download()[0], o.state()[0])


@pytest.mark.parametrize("mesh", ["hex", "tets", "symmetry", "constrained"])
@pytest.mark.parametrize("reconst", [cases.RECONST_NONE, cases.RECONST_WENO_SIMPLE, cases.RECONST_WENO_XYZ])
def test_gradients_by_variable_bit_exact(gpu_lib, mesh, reconst):
    """The unlimited gradient and the WENO smoothing by one thread per cell and
    variable, with reflected members, and beside constrained cells (which keep
    one thread per cell): FP64_EXACT equal to the oracle's bits."""
    num = cases.Numerics(space_order=2, space_discr=cases.DISCR_HLLC, reconst=reconst, cfl=0.4)
    if mesh == "tets":
        c = cases.adjoint_tets(4, num=num)
    elif mesh == "symmetry":
        c = cases.mirror_box(5, axes=(0, 1, 2), num=num)
    else:
        c = cases.shock_sphere(7, num=num)
        c.cv0 = _wavy(c)
    if mesh == "constrained":
        c.num.c_reconst = 1
    rhs_o, grad_o = Oracle(c).residual()
    rhs_g, grad_g = gpu.Region(c, "fp64_exact").residual(c.cv0)
    np.testing.assert_array_equal(grad_g, grad_o)
    np.testing.assert_array_equal(rhs_g, rhs_o)
