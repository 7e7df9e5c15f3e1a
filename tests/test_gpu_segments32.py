"""Segments of the mixed form (k_seg32): the bits of one launch per step.

The steps of a differentiated run go through the single-step kernels (k_step32
and its walk queue), which share the functions of push, walk and collision with
the segment kernel but not its groups and queues. The operations per particle
and step are the same, so the bar is identity of the final state, for every
segment length, at particle counts around a warp's group and beyond one block,
with sets that cross many tets, are slower than the reference's limit, do not
move, start outside the modelling box or the mesh, stop being numbers, or test
a collision in most steps.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _set(n, L, seed):
    rng = np.random.default_rng(seed)
    pos = rng.uniform(0.02 * L, 0.98 * L, (n, 3))
    vel = rng.normal(size=(n, 3)) * 4000.0
    kind = rng.integers(0, 24, n)
    vel[kind == 0] *= 1e-3                       # around the slow limit of 10 m/s
    vel[kind == 1] = 0.0                         # never moved (|v| below the limit)
    vel[kind == 2] *= 60.0                       # many tets in a step
    pos[kind == 3] = L * 1.5                     # outside the mesh: lost at once
    vel[(kind == 4) & (rng.random(n) < 0.3)] = np.inf  # the position stops being a number
    pos[kind == 5] = np.round(pos[kind == 5] / (L / 8)) * (L / 8)  # on lattice nodes
    return pos, vel


def _start(w, seg, pos, vel):
    from start_gb300 import StartPIC

    e = StartPIC(w.mesh, dict(w.params, precision=1))
    e.set_step_segments(seg)
    e.set_particles(pos, vel)
    e.set_potential(100.0 * np.sin(40.0 * w.mesh.nodes).sum(1))
    return e


@pytest.mark.parametrize("model,gas", [(0, 1.0), (1, 1.0), (1, 40.0), (2, 300.0), (3, 10.0)],
                         ids=["none", "hs", "hs_dense", "vhs_denser", "vss"])
@pytest.mark.parametrize("n", [1, 31, 33, 4000])
def test_same_bits_as_single_steps(built, n, model, gas):
    from start_gb300.workloads import workload0

    w = workload0(n_particles=1, cells=8, collisions=model != 0)
    w.params.update(collision_model=model, dt=2e-8, resort_every=0)
    w.params["gas_concentration"] *= gas
    pos, vel = _set(n, 0.1, seed=n + 7 * model)
    e = _start(w, 1, pos, vel)
    if model == 3:  # VSS has no differentiated run: one step per launch of the segment kernel
        e.process(70)
    else:
        e.grad_forward(70, (0.05, 0.05, 0.1), 0.01)
    ref = e.particles()
    e.close()
    for seg, calls in ((1, [70]), (7, [64, 6]), (32, [70]), (64, [64, 6])):
        e = _start(w, seg, pos, vel)
        for c in calls:
            st = e.process(c)
        got, tris = e.particles(), e.triangle_counts()
        e.close()
        for k in ("pos", "vel"):
            assert np.array_equal(got[k], ref[k], equal_nan=True), (seg, k)
        for k in ("tet", "flags"):
            assert np.array_equal(got[k], ref[k]), (seg, k)
        assert tris.sum() == st["n_settled"] == (got["flags"] & 1).sum()
        if n == 4000:
            assert st["crossings"] > 1000 and (model == 0) == (st["collisions"] == 0)


def test_lazy_field_many_warps_matches_full_field(built):
    """A run whose solves refresh only the occupied tets: fields formed during a
    segment, by several lanes at once, equal those of one launch per step."""
    from start_gb300 import StartPIC
    from start_gb300.workloads import workload1

    w = workload1(n_particles=300_000, cells=24)
    w.params.update(cg_rtol=1e-12, dt=2e-8, precision=1)
    out = []
    for seg in (1, 32):
        e = StartPIC(w.mesh, w.params)
        e.set_step_segments(seg)
        e.set_particles(w.pos, w.vel)
        st = e.run(60)
        p = e.particles()
        out.append((p["pos"], p["vel"], p["tet"], p["flags"], e.efield(), e.potential(),
                    np.array([st["crossings"], st["collisions"], st["n_settled"]])))
        e.close()
    for a, b in zip(*out):
        assert np.array_equal(a, b)
