"""The gradient when the particles change their order after the forward pass.

spg_resort, and steps that re-sort, put the particles into other slots; landings
and records stay in those of the forward pass. The backward pass replays the
collisions by particle id, so with the ids of another order it would replay
those of other particles. The dense gas makes that visible in every component.
Tolerance: the sums per tet in another order and the adjoint CG, stopped at
1e-13 of them: 1e-10 of the largest component; J, a sum of 3e3 terms in any
order, 1e-12.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _engine(precision, n=3000):
    from start_gb300 import StartPIC, mesh as M
    from start_gb300.workloads import TI_MASS, _base_params, gas_concentration

    L = 0.1
    m = M.kuhn_box((8, 8, 8), (L,) * 3)
    lo, hi = M.box_face_nodes(m, 2, 0), M.box_face_nodes(m, 2, 1)
    m.with_dirichlet(np.concatenate([lo, hi]), np.zeros(len(lo) + len(hi)))
    p = _base_params(dt=2e-8, weight=1e6, seed=5, collision_model=1, precision=precision, resort_every=0,
                     gas_concentration=gas_concentration(10.0, 300.0), cg_rtol=1e-13)
    e = StartPIC(m, p)
    g = np.zeros(m.n_nodes)
    g[hi] = 400.0
    e.set_dirichlet(g)
    e.set_particles(*_particles(n))
    e.solve(np.zeros(m.n_nodes), want_phi=False)
    return e


def _particles(n):
    from start_gb300.sources import make_particles
    from start_gb300.workloads import TI_MASS

    return make_particles(5, n, TI_MASS, source="disk", centre=(0.05, 0.05, 0.0), radius=0.02, directions="cone",
                          half_angle=0.5, energy="thompson")


@pytest.mark.parametrize("precision", [0, 1], ids=["fp64", "mixed"])
def test_resort_between_forward_and_backward(built, precision):
    out = []
    for between in ("nothing", "resort", "steps and resort"):
        e = _engine(precision)
        J, landed = e.grad_forward(120, np.array([0.05, 0.05, 0.0]), 0.02)
        if between != "nothing":
            if between != "resort":
                e.process(3)
            e.resort()
        out.append((J, landed, *e.grad_backward()[:3]))
        e.close()
    assert out[0][1] > 500 and all(np.abs(a).max() > 0 for a in out[0][2:])
    for got in out[1:]:
        assert got[1] == out[0][1] and abs(got[0] - out[0][0]) <= 1e-12 * abs(out[0][0])
        for a, b in zip(got[2:], out[0][2:]):
            assert np.abs(a - b).max() <= 1e-10 * np.abs(b).max()
