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


@pytest.mark.parametrize("mesh", ["hex", "tets", "periodic", "symmetry", "constrained"])
@pytest.mark.parametrize("state", ["wavy", "wide", "extreme", "still"])
def test_fixed_point_gradients(gpu_lib, mesh, state):
    """The least-squares sums of the fp64 mode in fixed point against the
    FP64_EXACT ones (unlimited gradients): values near each other, values
    spread over ten orders of magnitude, magnitudes outside the fixed point's
    range (the FP64 loop), a uniform state.  Bound: 1e-14 of the largest
    weight sum times the largest difference, per cell and variable."""
    num = cases.Numerics(space_order=2, space_discr=cases.DISCR_HLLC, reconst=cases.RECONST_NONE, cfl=0.4)
    if mesh == "tets":
        c = cases.adjoint_tets(4, num=num)
    elif mesh == "symmetry":
        c = cases.mirror_box(5, axes=(0, 1, 2), num=num)
    elif mesh == "periodic":
        c = cases.gas_jump_periodic(5)
        c.num.reconst = cases.RECONST_NONE
    else:
        c = cases.shock_sphere(7, num=num)
    if mesh == "constrained":
        c.num.c_reconst = 1
    rng = np.random.default_rng(9)
    n = len(c.cv0)
    rho, p = 1.0 + 0.3 * rng.random(n), 1.0 + 0.3 * rng.random(n)
    u = rng.standard_normal((n, 3))
    if state == "wide":
        rho, p = 10.0 ** rng.uniform(-5, 5, n), 10.0 ** rng.uniform(-5, 5, n)
        u = u * 10.0 ** rng.uniform(-8, 0, (n, 3))
    elif state == "extreme":
        u[::3, 0] *= 1e-160
        u[1::3, 1] = 1e-310
        u[:, 2] = 0.0
    elif state == "still":
        rho, p, u = np.ones(n), np.ones(n), np.zeros((n, 3))
    c.cv0 = cases.conserved(rho, u[:, 0], u[:, 1], u[:, 2], p, c.num.gamma)
    _, g = gpu.Region(c, "fp64").residual(c.cv0)
    _, ref = gpu.Region(c, "fp64_exact").residual(c.cv0)
    if state == "still":
        np.testing.assert_array_equal(g, 0.0)
        return
    # per variable the largest value over the smallest spacing of the mesh
    # bounds a cell's weights times differences; 40 members, FP64 rounding
    grid = gpu.Setup(c)
    h = grid.vol.min() ** (1 / 3)
    prim = np.stack([rho, u[:, 0], u[:, 1], u[:, 2], p], axis=1)
    scale = np.abs(prim).max(axis=0) / h
    assert (np.abs(g - ref).max(axis=2) / np.maximum(scale, 1e-300)).max() < 1e-14


@pytest.mark.parametrize("mesh", ["hex", "tets", "symmetry", "constrained", "periodic"])
@pytest.mark.parametrize("reconst", [cases.RECONST_NONE, cases.RECONST_BJ_COMP, cases.RECONST_VENKAT,
                                     cases.RECONST_BJ, cases.RECONST_WENO_XYZ])
def test_tangent_and_adjoint_of_the_fixed_sums(gpu_lib, mesh, reconst):
    """The fp64 mode's tangent (along the recorded branch) and adjoint against
    the FP64_EXACT mode's (dual numbers, FP64 sums): the same linear maps, to
    rounding amplified by the limiters' quotients."""
    num = cases.Numerics(space_order=2, space_discr=cases.DISCR_HLLC, reconst=reconst, cfl=0.4)
    if mesh == "tets":
        c = cases.adjoint_tets(4, num=num)
    elif mesh == "symmetry":
        c = cases.mirror_box(5, axes=(0, 1, 2), num=num)
    elif mesh == "periodic":
        c = cases.gas_jump_periodic(5, left=(1.2, 0.0, 1.0), right=(0.97, 0.8))
        c.num = num
    else:
        c = cases.shock_sphere(6, num=num)
    if mesh == "constrained":
        c.num.c_reconst = 1
    c.cv0 = _wavy(c, amp=0.02)
    rng = np.random.default_rng(2)
    dot, bar = rng.standard_normal(c.cv0.shape), rng.standard_normal(c.cv0.shape)
    a, b = gpu.Region(c, "fp64"), gpu.Region(c, "fp64_exact")
    for x, y in ((a.jvp(c.cv0, dot), b.jvp(c.cv0, dot)), (a.vjp(c.cv0, bar), b.vjp(c.cv0, bar))):
        assert np.isfinite(y).all()
        assert np.abs(x - y).max() <= 1e-9 * np.abs(y).max()


@pytest.mark.parametrize("order", [1, 2])
@pytest.mark.parametrize("discr", [cases.DISCR_ROE, cases.DISCR_HLLC, cases.DISCR_AUSM])
@pytest.mark.parametrize("mach", [0.0, 0.4, -2.5, 2.5])
def test_short_fluxes(gpu_lib, order, discr, mach):
    """The fp64 mode's interior fluxes against the FP64_EXACT ones, with the
    flow at rest, subsonic and supersonic either way: 1e-12 of each residual
    component's largest value."""
    num = cases.Numerics(space_order=order, space_discr=discr, reconst=0, cfl=0.4)
    c = cases.blast_hex(7, num=num)
    for p in c.patches:
        p.order = order
    rng = np.random.default_rng(8)
    n = len(c.cv0)
    rho, p = 1.0 + 0.2 * rng.random(n), 1.0 + 0.2 * rng.random(n)
    u = (mach * np.sqrt(1.4) + 0.05 * rng.standard_normal(n), 0.05 * rng.standard_normal(n), 0.05 * rng.standard_normal(n))
    c.cv0 = cases.conserved(rho, *u, p, c.num.gamma)
    a, _ = gpu.Region(c, "fp64").residual(c.cv0, with_grad=False)
    b, _ = gpu.Region(c, "fp64_exact").residual(c.cv0, with_grad=False)
    assert (np.abs(a - b) / np.abs(b).max(axis=0)).max() < 1e-12


@pytest.mark.parametrize("mesh", ["hex", "symmetry"])
@pytest.mark.parametrize("order", [1, 2])
@pytest.mark.parametrize("discr", [cases.DISCR_ROE, cases.DISCR_HLLC, cases.DISCR_AUSM])
@pytest.mark.parametrize("mach", [0.4, -2.5])
def test_short_flux_derivatives(gpu_lib, mesh, order, discr, mach):
    """Tangent and adjoint through the fp64 mode's fluxes (dual numbers over
    the short form, normals without derivatives) against the FP64_EXACT ones,
    unlimited gradients: 1e-11 of the largest value, some 500 roundings with
    room for their cancellation."""
    num = cases.Numerics(space_order=order, space_discr=discr, reconst=0, cfl=0.4)
    c = cases.mirror_box(5, axes=(0, 1, 2), num=num) if mesh == "symmetry" else cases.blast_hex(6, num=num)
    for p in c.patches:
        p.order = order
    rng = np.random.default_rng(9)
    n = len(c.cv0)
    rho, p = 1.0 + 0.2 * rng.random(n), 1.0 + 0.2 * rng.random(n)
    u = (mach * np.sqrt(1.4) + 0.05 * rng.standard_normal(n), 0.05 * rng.standard_normal(n), 0.05 * rng.standard_normal(n))
    c.cv0 = cases.conserved(rho, *u, p, c.num.gamma)
    dot, bar = rng.standard_normal(c.cv0.shape), rng.standard_normal(c.cv0.shape)
    a, b = gpu.Region(c, "fp64"), gpu.Region(c, "fp64_exact")
    for x, y in ((a.jvp(c.cv0, dot), b.jvp(c.cv0, dot)), (a.vjp(c.cv0, bar), b.vjp(c.cv0, bar))):
        assert np.isfinite(y).all()
        assert np.abs(x - y).max() <= 1e-11 * np.abs(y).max()


@pytest.mark.parametrize("mesh", ["hex", "tets", "symmetry", "periodic"])
@pytest.mark.parametrize("reconst", [cases.RECONST_BJ, cases.RECONST_BJ_COMP])
@pytest.mark.parametrize("flow", ["wavy", "shear", "still", "steep", "small"])
def test_limiter_in_one_pass(gpu_lib, mesh, reconst, flow):
    """The fp64 mode's Barth-Jespersen limiters (one pass over the faces, the
    frame by FP32 rotations first) against the FP64_EXACT ones: three-
    dimensional gradients, a shear with a repeated strain eigenvalue, none,
    1e6 jumps and differences of 1e-9.  1e-10 of a variable's largest
    gradient: the frame's tolerance (1e-12) over the eigenvalue gaps the
    limiter does not merge (1e-3), with room for the FP64 sums' rounding."""
    num = cases.Numerics(space_order=2, space_discr=cases.DISCR_HLLC, reconst=reconst, cfl=0.4)
    if mesh == "tets":
        c = cases.adjoint_tets(4, num=num)
    elif mesh == "symmetry":
        c = cases.mirror_box(5, axes=(0, 1, 2), num=num)
    elif mesh == "periodic":
        c = cases.gas_jump_periodic(5, length=1.0, x_jump=0.5)
        c.num = num
    else:
        c = cases.shock_sphere(7, num=num)
    rng = np.random.default_rng(12)
    n, x = len(c.cv0), gpu.Setup(c).cofg
    rho, p, u = np.ones(n), np.ones(n), np.zeros((n, 3))
    if flow in ("wavy", "small"):
        amp = 1e-9 if flow == "small" else 0.2
        rho, p = 1.0 + amp * rng.random(n), 1.0 + amp * rng.random(n)
        u = amp * rng.standard_normal((n, 3))
    elif flow == "shear":
        u[:, 0] = np.sin(3 * x[:, 1])
        u[:, 1] = 0.3 * np.sin(3 * x[:, 1] + 0.4)
        u[:, 2] = 0.2 * np.cos(2 * x[:, 1] + x[:, 0])
    elif flow == "steep":
        rho, p = np.where(x[:, 0] < 0.5, 1e6, 1.0) * (1 + 0.1 * rng.random(n)), np.where(x[:, 1] < 0.5, 1e6, 1.0)
        u = rng.standard_normal((n, 3)) * np.where(x[:, 2:] < 0.5, 1e3, 1e-3)
    c.cv0 = cases.conserved(rho, u[:, 0], u[:, 1], u[:, 2], p, c.num.gamma)
    _, a = gpu.Region(c, "fp64").residual(c.cv0)
    _, b = gpu.Region(c, "fp64_exact").residual(c.cv0)
    top = np.abs(b).max(axis=(0, 2))
    if reconst == cases.RECONST_BJ:
        top[1:4] = top[1:4].max()  # the frame mixes the components
    # a uniform variable's gradient is the rounding of its values over the spacing
    # (the pressure's, of the total energy it is recovered from)
    prim = np.abs(np.stack([rho, u[:, 0], u[:, 1], u[:, 2], c.cv0[:, 4]], axis=1)).max(axis=0)
    floor = 1e-14 * prim / gpu.Setup(c).vol.min() ** (1 / 3)
    assert (np.abs(a - b).max(axis=(0, 2)) <= 1e-10 * top + floor).all(), (np.abs(a - b).max(axis=(0, 2)), top)


@pytest.mark.parametrize("rho0", [1.0, 1e-35])
@pytest.mark.parametrize("p0", [1e-12, 1e-2])
@pytest.mark.parametrize("cfl", [1, 3])
def test_bounds_check_only_near_zero(gpu_lib, rho0, p0, cfl):
    """Still gas overdriven to pressures either side of zero, inside and
    outside the 1e-12 of the bounds check and inside and outside the range in
    which the update skips it: counters and bits of the oracle."""
    c = cases.sod(40, 1, 1)
    c.num.rk_scheme = cases.RK_EULER
    rng = np.random.default_rng(4)
    n = len(c.cv0)
    p, rho, z = p0 * 2 * rng.random(n), rho0 * (1 + 0.5 * rng.random(n)), np.zeros(n)
    c.cv0 = cases.conserved(rho, z, z, z, p, 1.4)
    dt = cfl * 0.025 / np.sqrt(1.4 * p0 / rho0)
    o = Oracle(c)
    o.rk_stage(1, dt)
    pf, neg, nan = o.counters()
    assert nan == 0 and (pf > 0) == (cfl == 3) and (neg > 0) == (cfl == 3 and p0 == 1e-12)
    r = gpu.Region(c, "fp64_exact")
    r.rk_stage(1, dt)
    st = r.status()
    assert (st["posFixCells"], st["negPCells"], st["nanCells"]) == (pf, neg, nan)
    np.testing.assert_array_equal(r.download()[0], o.state()[0])
