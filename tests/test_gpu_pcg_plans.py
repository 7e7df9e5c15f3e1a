"""Several launch plans of the one-launch Jacobi PCG alive at once.

The solver's kernels serve plans of very different shared memory (a block of 512
threads needs four times that of 128), and a plan outlives the call that made
it: in a handle, and for the last row count of spg_pcg_solve_noalloc. Making one
must not change what another one may launch with. Every solve is checked by its
own residual b - K phi in NumPy, within twice the stop tolerance.
"""
import ctypes as C

import numpy as np
import pytest

from test_gpu_pcg_resident import RTOL, _system

pytestmark = pytest.mark.gpu

# 68,921 and 29,791 (512 and 256 threads a block), 17,576 (128), 4,913 (128, few blocks), and the
# cluster form's largest and a small one: 4,096 and 1,331
CELLS = [40, 30, 25, 16, 15, 10]


class _Handle:
    def __init__(self, cells):
        from start_gb300 import StartPIC, mesh as M
        from start_gb300.workloads import EPS0, _base_params, _zbc

        self.m = _zbc(M.kuhn_box((cells,) * 3, (0.1,) * 3))
        self.eng = StartPIC(self.m, _base_params(cg_rtol=1e-10))
        rp, col, self.val, self.lift, dual = self.eng.matrix()
        self.rp, self.col, self.scale = rp, col, dual / EPS0
        self.rng = np.random.default_rng(cells)

    def solve(self):
        rho = self.rng.uniform(0.0, 1e-7, self.m.n_nodes)
        phi, it, rr = self.eng.solve(rho)
        b = rho * self.scale - self.lift
        b[self.m.dirichlet_nodes] = self.m.dirichlet_values
        r = b - np.add.reduceat(self.val * phi[self.col], self.rp[:-1])
        assert it > 5 and rr <= 1e-10
        assert np.linalg.norm(r) <= 2e-10 * np.linalg.norm(b)


@pytest.mark.parametrize("order", [1, -1], ids=["largest_first", "smallest_first"])
def test_handles_of_many_sizes_solve_side_by_side(built, order):
    hs = [_Handle(c) for c in CELLS[::order]]
    for h in hs + hs[::-1]:
        h.solve()
    for h in hs:
        h.eng.close()


def _noalloc(n, couplings):
    import torch

    from start_gb300 import _native as N

    lib = N.load()
    rp, col, val, b, x = _system(n, couplings, seed=n)
    dev = [torch.from_numpy(a).cuda() for a in (rp, col, val, b, np.zeros(n))]

    def solve():
        dev[4].zero_()
        torch.cuda.synchronize()
        it, rr = C.c_int32(), C.c_double()
        rc = lib.spg_pcg_solve_noalloc(n, *[a.data_ptr() for a in dev], RTOL, 500, None, C.byref(it), C.byref(rr))
        assert rc == 0, lib.spg_last_error(None).decode()
        assert np.linalg.norm(dev[4].cpu().numpy() - x) <= 2.0 * RTOL * np.linalg.norm(b)

    return solve


def test_handles_made_between_allocation_free_solves(built):
    large, small = _noalloc(70_000, 6), _noalloc(3_000, 6)
    # both sides of the cluster form's limit, rows in random order, more couplings than are staged
    edges = [_noalloc(4096, 40), _noalloc(4097, 40)]
    a = _Handle(40)
    large()
    b, c = _Handle(16), _Handle(10)
    large()  # the same row count as before: its plan is kept
    small()
    large()
    for h in (a, c, b, a):
        h.solve()
    for s in edges + [small, large]:
        s()
    for h in (a, b, c):
        h.eng.close()
