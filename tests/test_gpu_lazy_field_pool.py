"""Fields formed during a segment, read by particles that come back from a pool.

A particle that enters a tet whose field is of an older potential forms that
field itself, while another lane, of any warp, may be storing it. When the
particle then waits for a collision test, or for a walk that ends where it began,
it has to form the field again: the stores of its own launch are ordered with
nothing. In a gas so dense that most steps test a collision, with many particles
per tet and solves that refresh the occupied tets only, every segment does this
many times. Launches of one step never read a field of their own launch, and the
operations per particle are the same, so the bar is identity.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", [0, 1], ids=["fp64", "mixed"])
@pytest.mark.parametrize("cells,n", [(8, 300_000), (24, 100_000)])
def test_pooled_particles_form_the_field_of_their_tet(built, cells, n, precision):
    from start_gb300 import StartPIC
    from start_gb300.workloads import workload1

    w = workload1(n_particles=n, cells=cells)
    w.params.update(cg_rtol=1e-12, dt=2e-7, precision=precision, collision_model=1)
    w.params["gas_concentration"] *= 3.0
    out = []
    for seg in (1, 64):
        e = StartPIC(w.mesh, w.params)
        e.set_step_segments(seg)
        e.set_particles(w.pos, w.vel)
        st = e.run(40)
        p = e.particles()
        out.append((p["pos"], p["vel"], p["tet"], p["flags"], e.efield(), e.potential(),
                    np.array([st["crossings"], st["collisions"], st["n_settled"]])))
        e.close()
    assert out[0][6][0] > n / 10 and out[0][6][1] > n  # tets are entered, and collisions are many
    for a, b in zip(*out):
        assert np.array_equal(a, b)
