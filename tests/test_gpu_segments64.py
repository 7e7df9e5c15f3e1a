"""Segments of the FP64 form (k_seg64): the same bits for every segment length
and every particle count.

The operations per particle and step do not depend on how many steps a launch
takes, on the warp that runs the particle or on the pool it passes through, so
the bar is identity. Counts sit at the edges of a warp's batches (one lane, one
warp, one more) and beyond one wave; the sets hold particles that cross many
tets, that are slower than the reference's limit, that do not move, that start
outside the modelling box or the mesh, and positions that stop being numbers.
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
    vel[kind == 3] = rng.normal(size=((kind == 3).sum(), 3)) * 1e-30 + np.array([20.0, 0.0, 0.0])
    pos[kind == 4] = L * 1.5                     # outside the mesh: lost at once
    vel[(kind == 5) & (rng.random(n) < 0.3)] = np.inf  # the position stops being a number
    pos[kind == 6] = np.round(pos[kind == 6] / (L / 8)) * (L / 8)  # on lattice nodes
    return pos, vel


def _run(w, n, seg, pos, vel, calls):
    from start_gb300 import StartPIC

    e = StartPIC(w.mesh, w.params)
    e.set_step_segments(seg)
    e.set_particles(pos, vel)
    phi = 100.0 * np.sin(40.0 * w.mesh.nodes).sum(1)
    e.set_potential(phi)
    for c in calls:
        st = e.process(c)
    p = e.particles()
    out = (p["pos"], p["vel"], p["tet"], p["flags"], e.triangle_counts(),
           np.array([st[k] for k in ("n_alive", "n_settled", "n_lost", "particle_steps", "collisions", "crossings")]))
    e.close()
    return out


@pytest.mark.parametrize("model,gas", [(0, 1.0), (1, 1.0), (1, 40.0), (2, 10.0), (3, 10.0)],
                         ids=["none", "hs", "hs_dense", "vhs", "vss"])
@pytest.mark.parametrize("n", [1, 31, 33, 4000])
def test_same_bits_for_every_segment(built, n, model, gas):
    from start_gb300.workloads import workload0

    w = workload0(n_particles=1, cells=8, collisions=model != 0)
    w.params.update(collision_model=model, dt=2e-8, resort_every=0)
    w.params["gas_concentration"] *= gas
    pos, vel = _set(n, 0.1, seed=n + 7 * model)
    ref = _run(w, n, 1, pos, vel, [64, 6])
    for seg, calls in ((7, [64, 6]), (32, [70]), (64, [64, 6])):
        got = _run(w, n, seg, pos, vel, calls)
        for a, b in zip(ref, got):
            assert np.array_equal(a, b, equal_nan=a.dtype.kind == "f")
    if n == 4000:
        assert ref[5][5] > 1000 and (model == 0) == (ref[5][4] == 0)


def test_lazy_field_many_warps_matches_single_steps(built):
    """A run whose solves refresh only the occupied tets: fields formed during a
    segment (by several lanes at once) equal those of one launch per step."""
    from start_gb300 import StartPIC
    from start_gb300.workloads import workload1

    w = workload1(n_particles=300_000, cells=24)
    w.params.update(cg_rtol=1e-12, dt=2e-8)
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
