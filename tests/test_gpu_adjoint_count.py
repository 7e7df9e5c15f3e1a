"""The gradient after the particle set was replaced by one of another size.

Landings, records and results are sized for the particles of the forward pass,
so the backward pass refuses another count.
"""
import numpy as np
import pytest

from test_gpu_adjoint_order import _engine, _particles

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", [0, 1], ids=["fp64", "mixed"])
@pytest.mark.parametrize("how", ["set_particles", "restore"])
def test_another_particle_count_is_refused(built, precision, how):
    from start_gb300.engine import PICBaseException

    e = _engine(precision, 500)
    if how == "restore":
        blob = e.checkpoint()
        e.set_particles(*_particles(3000))
        e.solve(np.zeros(e.mesh.n_nodes), want_phi=False)
    _, landed = e.grad_forward(120, np.array([0.05, 0.05, 0.0]), 0.02)
    assert landed > 50
    if how == "restore":
        e.restore(blob)
    else:
        e.set_particles(*_particles(3000))
    with pytest.raises(PICBaseException, match="grad_forward"):
        e.grad_backward()
    e.close()
