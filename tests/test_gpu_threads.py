"""Contexts in several host threads."""
import threading

import numpy as np
import pytest

from rocflu_gb300 import cases, gpu

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_adjoints_in_two_threads(gpu_lib, precision):
    """Two threads' VJPs, each on a context of its own with boundary faces (the
    boundary kernel runs beside the interior one on a second stream): the same
    bits as one after the other."""
    num = cases.Numerics(space_order=2, space_discr=cases.DISCR_HLLC, reconst=cases.RECONST_BJ_COMP, cfl=0.4)
    work = []
    for n in (12, 17):
        c = cases.blast_hex(n, num=num)
        rng = np.random.default_rng(n)
        c.cv0 = c.cv0 * (1.0 + 0.01 * rng.standard_normal(c.cv0.shape))
        bars = rng.standard_normal((20,) + c.cv0.shape)
        r = gpu.Region(c, precision)
        work.append((r, c.cv0, bars, [r.vjp(c.cv0, b) for b in bars]))
    got = [[None] * 20 for _ in work]

    def run(k):
        r, cv, bars, _ = work[k]
        for m, b in enumerate(bars):
            got[k][m] = r.vjp(cv, b)

    team = [threading.Thread(target=run, args=(k,)) for k in range(2)]
    for t in team:
        t.start()
    for t in team:
        t.join()
    for k, (_, _, _, want) in enumerate(work):
        for a, b in zip(got[k], want):
            np.testing.assert_array_equal(a, b)


def test_contexts_made_in_two_threads(gpu_lib):
    """Tiled contexts of a small and a larger mesh made at the same time, eight
    times: both run (the kernels' shared memory limit is the larger one's)."""
    num = cases.Numerics(space_order=2, space_discr=cases.DISCR_HLLC, reconst=cases.RECONST_BJ, cfl=0.4)
    meshes = [cases.shock_sphere(6, num=num), cases.blast_tets(10, num=num)]
    grids = [gpu.Setup(c) for c in meshes]
    want = []
    for c, g in zip(meshes, grids):
        r = gpu.Region(c, "mixed", grid=g)
        r.run_fixed_dt(2, 1e-5)
        want.append(r.download()[0])
    got, wrong = [[], []], []

    def run(k, gate):
        try:
            gate.wait()
            r = gpu.Region(meshes[k], "mixed", grid=grids[k])
            r.run_fixed_dt(2, 1e-5)
            got[k].append(r.download()[0])
        except Exception as e:  # noqa: BLE001 - reported by the test's own thread
            wrong.append(e)

    for _ in range(8):
        gate = threading.Barrier(2)
        team = [threading.Thread(target=run, args=(k, gate)) for k in range(2)]
        for t in team:
            t.start()
        for t in team:
            t.join()
    assert not wrong, wrong[0]
    for k in range(2):
        assert len(got[k]) == 8
        for x in got[k]:
            np.testing.assert_array_equal(x, want[k])
