"""The adjoint from the forward's own record of every step, against the windows
that are repeated from checkpoints when the record does not fit.

Without collisions the particles are independent and alike, so a set of 400
(recorded) and the same 400 repeated 2,500 times (1e6 particles, 2,400 steps: 77
GB, more than the record may take) have the same J and dJ/dg, and 2,500 times
the derivative of each particle. The sums over particles are of 1e6 FP64 terms in
another order: 1e-10 of the largest component covers them; a second backward pass
of the record returns what the first did, up to the order of the same sums.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

STEPS, FEW, TIMES = 2400, 400, 2500


def _grads(pos, vel, passes):
    from start_gb300 import StartPIC
    from start_gb300.workloads import workload0

    w = workload0(n_particles=1, cells=8, collisions=False)
    w.params.update(resort_every=0, cg_rtol=1e-12, dt=2e-9)
    e = StartPIC(w.mesh, w.params)
    e.set_particles(pos, vel)
    e.solve(np.zeros(w.mesh.n_nodes), want_phi=False)
    J, landed = e.grad_forward(STEPS, (0.05, 0.05, 0.1), 0.01)
    out = [(J, landed, *e.grad_backward()[:3]) for _ in range(passes)]
    e.close()
    return out


def test_record_and_windows_agree(built):
    rng = np.random.default_rng(2)
    pos = rng.uniform(0.03, 0.07, (FEW, 3))
    vel = rng.normal(size=(FEW, 3)) * 3000.0 + np.array([0.0, 0.0, 6000.0])
    (a, b), (c,) = _grads(pos, vel, 2), _grads(np.tile(pos, (TIMES, 1)), np.tile(vel, (TIMES, 1)), 1)
    assert a[1] > 0 and c[1] == a[1] * TIMES  # (8 of the 400 land)
    assert abs(c[0] - a[0]) <= 1e-12 * abs(a[0])
    for x, y in zip(a[2:], b[2:]):
        assert np.abs(x - y).max() <= 1e-10 * np.abs(x).max()
    assert np.abs(c[2] - a[2]).max() <= 1e-10 * np.abs(a[2]).max()
    for k in (3, 4):
        got = c[k].reshape(TIMES, FEW, 3) * TIMES
        assert np.abs(got - a[k]).max() <= 1e-10 * np.abs(a[k]).max()
