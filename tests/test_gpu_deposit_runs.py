"""The deposit at the edges of its tiles and runs, against weights in NumPy.

Particles in an order that makes one run of equal tets per warp, two tets
alternating from lane to lane (32 runs, every add of a block to the same two
slots of its table: carries between the halves of a sum), and random tets.
Node charges in particles: each FP64 weight is off by its fixed-point rounding
(2^-40 at these counts at most) and a few eps, so n particles by at most 2e-12
n; in the mixed form the FP32 local position and map put a weight within 2e-6.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _points(m, tets, rng):
    lam = rng.dirichlet(np.ones(4), len(tets))
    return np.einsum("ij,ijk->ik", 0.9 * lam + 0.025, m.nodes[m.tets[tets]])


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("order", ["one", "alternate", "random"])
@pytest.mark.parametrize("n", [1, 31, 33, 255, 257, 4096, 70001])
def test_node_charges(built, n, order, precision):
    from start_gb300 import StartPIC
    from start_gb300 import mesh as M
    from start_gb300.workloads import _base_params, _zbc

    m = _zbc(M.kuhn_box((6, 5, 4), (0.06, 0.05, 0.04)))
    rng = np.random.default_rng(n)
    pick = {"one": np.full(n, 100), "alternate": np.where(np.arange(n) % 2, 100, 501),
            "random": rng.integers(0, m.n_tets, n)}[order]
    pos = _points(m, pick, rng)
    e = StartPIC(m, _base_params(precision=precision, resort_every=0))
    e.set_particles(pos, np.zeros((n, 3)))
    assert np.array_equal(e.particles()["tet"], pick)
    rho = e.gather()
    p = e.params if isinstance(getattr(e, "params", None), dict) else _base_params()
    e.close()
    dual = np.zeros(m.n_nodes)
    np.add.at(dual, m.tets.ravel(), np.repeat(m.volumes() / 4.0, 4))
    x = m.nodes[m.tets[pick]]
    J = np.stack([x[:, 1] - x[:, 0], x[:, 2] - x[:, 0], x[:, 3] - x[:, 0]], axis=2)
    l = np.linalg.solve(J, (pos - x[:, 0])[:, :, None])[:, :, 0]
    l = np.concatenate([1.0 - l.sum(1, keepdims=True), l], axis=1)
    want = np.zeros(m.n_nodes)
    np.add.at(want, m.tets[pick].ravel(), l.ravel())
    got = rho * dual / (p["charge"] * p["weight"])
    assert np.abs(got - want).max() <= n * (2e-12 if precision == 0 else 2e-6) + 1e-12 * n
    # every particle's four weights sum to one unit exactly
    assert abs(got.sum() - n) <= 1e-12 * n
