"""Solves whose matrix is stored with banded slices (nodes numbered along
lines) and without (the same mesh with its nodes renumbered at random).

Zero density between plates at 0 and 100 V: the P1 potential is 100 z / L
exactly. With cubic cells of size h each line of nodes along z carries at least
a quarter of h times the path's Laplacian, so lambda_min(A) >= h sin^2(pi / (2
nz)), and with ||b|| <= 101 sqrt(nodes of a plate) the solve's ||r|| <= rtol
||b|| bounds the error; 1.1 covers the difference of the recursive residual
from the true one (about 100 eps ||A|| ||phi||, below 0.01 rtol ||b||). The
V-cycle only steers the iterations, so their count is held too: the two
numberings aggregate differently, within half as many again and three.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

RTOL = 1e-12
H = 0.01


def _mesh(cells, lines):
    from start_gb300 import mesh as M
    from start_gb300.workloads import _zbc

    m = _zbc(M.kuhn_box(cells, tuple(H * c for c in cells)))
    if not lines:
        new = np.random.default_rng(3).permutation(m.n_nodes).astype(np.int32)
        nodes = np.empty_like(m.nodes)
        nodes[new] = m.nodes
        m.nodes, m.tets, m.triangles = nodes, new[m.tets], new[m.triangles]
        m.with_dirichlet(new[m.dirichlet_nodes], m.dirichlet_values)
    return m


# lines of 32, 33, 101 and 10 nodes; the last one above the one-launch Jacobi PCG
@pytest.mark.parametrize("precond", [0, 1, 2])
@pytest.mark.parametrize("cells", [(31, 12, 9), (32, 11, 10), (100, 9, 8), (9, 20, 21), (57, 54, 51)])
def test_linear_potential_in_both_numberings(built, cells, precond):
    from start_gb300 import StartPIC
    from start_gb300.workloads import _base_params

    its = []
    for lines in (True, False):
        m = _mesh(cells, lines)
        e = StartPIC(m, _base_params(cg_rtol=RTOL, preconditioner=precond))
        start = np.zeros(m.n_nodes)
        start[m.dirichlet_nodes] = m.dirichlet_values
        e.set_potential(start)
        phi, it, relres = e.solve(np.zeros(m.n_nodes))
        e.close()
        its.append(it)
        assert relres <= RTOL
        exact = 100.0 * m.nodes[:, 2] / (H * cells[2])
        plate = (cells[0] + 1) * (cells[1] + 1)
        bound = 1.1 * RTOL * 101.0 * np.sqrt(plate) / (H * np.sin(np.pi / (2 * cells[2])) ** 2)
        assert np.linalg.norm(phi - exact) <= bound, (lines, np.linalg.norm(phi - exact), bound)
    assert max(its) <= 1.5 * min(its) + 3, its
