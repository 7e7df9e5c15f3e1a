"""The adjoint's checkpoint windows and its collision screens on the GPU.

dJ/dx0, dJ/dv0 and dJ/dg do not depend on where the checkpoints lie: windows of
1, 7, 32, 100 (more than a segment) and all steps give the same gradients up to
the order of the per-tet sums. The gas is dense enough that a step's collision
probability lies on both sides of 1/256, so every branch of the backward pass's
screen decides, and a particle set with slow and lost ions is among them.
Tolerance: the sums of at most 2e3 terms per tet in another order, and the
adjoint CG stopped at 1e-13 of them: 1e-10 of the largest component.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _gradients(model, precision, every, gas):
    from start_gb300 import StartPIC, mesh as M
    from start_gb300.sources import make_particles
    from start_gb300.workloads import TI_MASS, _base_params, gas_concentration

    L = 0.1
    m = M.kuhn_box((8, 8, 8), (L,) * 3)
    lo, hi = M.box_face_nodes(m, 2, 0), M.box_face_nodes(m, 2, 1)
    m.with_dirichlet(np.concatenate([lo, hi]), np.zeros(len(lo) + len(hi)))
    p = _base_params(dt=2e-8, weight=1e6, seed=5, collision_model=model, precision=precision, resort_every=0,
                     gas_concentration=gas_concentration(gas, 300.0), cg_rtol=1e-13)
    pos, vel = make_particles(5, 2000, TI_MASS, source="disk", centre=(L / 2, L / 2, 0.0), radius=0.02,
                              directions="cone", half_angle=0.5, energy="thompson")
    vel[::97] *= 1e-4
    pos[::501] = 2 * L
    e = StartPIC(m, p)
    g = np.zeros(m.n_nodes)
    g[hi] = 400.0
    e.set_dirichlet(g)
    e.set_particles(pos, vel)
    e.solve(np.zeros(m.n_nodes), want_phi=False)
    J, landed = e.grad_forward(120, np.array([L / 2, L / 2, 0.0]), 0.02, checkpoint_every=every)
    dg, dx, dv, _ = e.grad_backward()
    e.close()
    return J, landed, dg, dx, dv


@pytest.mark.parametrize("precision", [0, 1], ids=["fp64", "mixed"])
@pytest.mark.parametrize("model,gas", [(0, 1.0), (1, 10.0), (2, 40.0)], ids=["none", "hs", "vhs"])
def test_gradient_does_not_depend_on_the_windows(built, model, gas, precision):
    ref = _gradients(model, precision, 120, gas)
    assert ref[1] > 500 and all(np.abs(a).max() > 0 for a in ref[2:])
    for every in (1, 7, 32, 100):
        got = _gradients(model, precision, every, gas)
        assert got[1] == ref[1] and abs(got[0] - ref[0]) <= 1e-12 * abs(ref[0])
        for a, b in zip(got[2:], ref[2:]):
            assert np.abs(a - b).max() <= 1e-10 * np.abs(b).max()
