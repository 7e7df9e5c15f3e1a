"""The re-sort of a new particle set (ranks and records) around the size from
which it is taken, with particles spread over all tets, sharing a few of them in
any order, and outside the mesh; then a later re-sort of the same handle.

A re-sort changes only the memory order: the particles by id are the same bits
before and after, and the deposit, whose integer sums do not depend on the
order, equals that of a handle that never sorts.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("where", ["spread", "few"])
@pytest.mark.parametrize("n", [65535, 65536, 65537, 100003])
def test_same_particles_after_a_sort(built, n, where, precision):
    from start_gb300 import StartPIC
    from start_gb300 import mesh as M
    from start_gb300.workloads import _base_params, _zbc

    m = _zbc(M.kuhn_box((12, 11, 10), (0.12, 0.11, 0.1)))
    rng = np.random.default_rng(n)
    pos = rng.uniform(0.001, 0.099, (n, 3))
    if where == "few":
        pos = 0.05 + 0.012 * (pos / 0.1)
    pos[rng.random(n) < 0.02] = 0.5  # outside the mesh
    vel = rng.normal(size=(n, 3)) * 3000.0
    out = []
    for every in (20, 0):
        e = StartPIC(m, _base_params(precision=precision, resort_every=every, dt=2e-8))
        for again in range(2):  # the second set reuses the records
            e.set_particles(pos, vel)
            before = e.particles()
            rho = e.gather()
            after = e.particles()
            for k in ("pos", "vel", "tet", "flags"):
                assert np.array_equal(before[k], after[k], equal_nan=True), (every, again, k)
        e.process(20)
        rho2 = e.gather()  # a later re-sort
        out.append((rho, rho2, *(e.particles()[k] for k in ("pos", "vel", "tet", "flags"))))
        e.close()
    for a, b in zip(*out):
        assert np.array_equal(a, b)
