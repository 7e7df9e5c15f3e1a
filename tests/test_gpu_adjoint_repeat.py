"""The FP64 gradient from checkpoint windows against the one from the record.

With the record's limit at zero the forward pass keeps checkpoints and the
backward pass repeats the steps of each window, whatever memory is free: the
same landings, J and gradients as from the forward's own record of every step,
for windows of 1, 7, 32, 100 (more than a segment) and all steps, without
collisions and in gases whose collision probability per step lies on both sides
of 1/256, with slow and lost ions among the particles. Tolerance: the sums of at
most 2e3 terms per tet in another order, and the adjoint CG stopped at 1e-13 of
them: 1e-10 of the largest component; J 1e-12.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

L, N, STEPS = 0.1, 2000, 120


def _engine(model, gas):
    from start_gb300 import StartPIC, mesh as M
    from start_gb300.sources import make_particles
    from start_gb300.workloads import TI_MASS, _base_params, gas_concentration

    m = M.kuhn_box((8, 8, 8), (L,) * 3)
    lo, hi = M.box_face_nodes(m, 2, 0), M.box_face_nodes(m, 2, 1)
    m.with_dirichlet(np.concatenate([lo, hi]), np.zeros(len(lo) + len(hi)))
    p = _base_params(dt=2e-8, weight=1e6, seed=5, collision_model=model, resort_every=0,
                     gas_concentration=gas_concentration(gas, 300.0), cg_rtol=1e-13)
    pos, vel = make_particles(5, N, TI_MASS, source="disk", centre=(L / 2, L / 2, 0.0), radius=0.02,
                              directions="cone", half_angle=0.5, energy="thompson")
    vel[::97] *= 1e-4
    pos[::501] = 2 * L
    e = StartPIC(m, p)
    g = np.zeros(m.n_nodes)
    g[hi] = 400.0
    e.set_dirichlet(g)
    e.start = pos, vel
    _restart(e)
    return e


def _restart(e):
    e.set_particles(*e.start)
    e.solve(np.zeros(e.n_nodes), want_phi=False)


def _forward(e, every=32):
    return e.grad_forward(STEPS, np.array([L / 2, L / 2, 0.0]), 0.02, checkpoint_every=every)


def _same(got, ref):
    assert got[1] == ref[1] and abs(got[0] - ref[0]) <= 1e-12 * abs(ref[0])
    for a, b in zip(got[2:], ref[2:]):
        assert np.abs(a - b).max() <= 1e-10 * np.abs(b).max()


@pytest.mark.parametrize("model,gas", [(0, 1.0), (1, 10.0), (2, 40.0)], ids=["none", "hs", "vhs"])
def test_windows_equal_the_record(built, model, gas):
    e = _engine(model, gas)
    ref = (*_forward(e), *e.grad_backward()[:3])
    e.close()
    assert ref[1] > 500 and all(np.abs(a).max() > 0 for a in ref[2:])
    for every in (1, 7, 32, 100, STEPS):
        e = _engine(model, gas)
        e.set_grad_record(0)
        got = (*_forward(e, every), *e.grad_backward()[:3])
        _same(got, ref)
        if every == 32:
            e.resort()  # ids and slots are those of the forward pass here too
            _same((*got[:2], *e.grad_backward()[:3]), ref)
        e.close()


def test_a_record_above_the_limit_is_given_back(built):
    from start_gb300.engine import PICBaseException

    e = _engine(1, 10.0)
    ref = (*_forward(e), *e.grad_backward()[:3])
    e.set_grad_record(32 * N * (STEPS + 2))  # the record just fits
    _same((*ref[:2], *e.grad_backward()[:3]), ref)
    e.set_grad_record(32 * N * (STEPS + 2) - 1)
    with pytest.raises(PICBaseException, match="grad_forward"):
        e.grad_backward()
    _restart(e)
    _same((*_forward(e), *e.grad_backward()[:3]), ref)  # the windows
    e.set_grad_record(1 << 35)
    _restart(e)
    _same((*_forward(e), *e.grad_backward()[:3]), ref)
    e.close()
