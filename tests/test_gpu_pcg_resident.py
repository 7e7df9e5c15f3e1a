"""The one-launch Jacobi PCG (kernels_pcg_resident.cu) at the edges of its launch shapes.

Systems with a known solution: A symmetric, a_ii = 1 + 1.5 sum |a_ij|, so by
Gershgorin the smallest eigenvalue is at least 1 and ||x - x*|| <= ||b - A x||
<= rtol ||b||. The bound tested is twice that: the recurrence residual the
solve stops on and the rounding of b = A x* each differ from the true residual
by a few hundred eps ||b||, far below rtol = 1e-11.
"""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

RTOL = 1e-11


def _system(n, couplings, seed):
    """Random symmetric couplings (some explicit zeros), rows in random column order, CSR."""
    rng = np.random.default_rng(seed)
    m = n * couplings // 2
    i, j = rng.integers(0, n, m), rng.integers(0, n, m)
    i, j = i[i != j], j[i != j]
    key = np.unique(np.minimum(i, j) * n + np.maximum(i, j))
    i, j = key // n, key % n
    v = rng.uniform(-1.0, 1.0, len(i))
    v[rng.random(len(i)) < 0.1] = 0.0
    diag = np.full(n, 1.0)
    np.add.at(diag, i, 1.5 * np.abs(v))
    np.add.at(diag, j, 1.5 * np.abs(v))
    row = np.concatenate([i, j, np.arange(n)])
    col = np.concatenate([j, i, np.arange(n)])
    val = np.concatenate([v, v, diag])
    order = np.lexsort((rng.random(len(row)), row))
    row, col, val = row[order], col[order], val[order]
    rp = np.concatenate([[0], np.cumsum(np.bincount(row, minlength=n))])
    x = rng.normal(size=n)
    b = np.bincount(row, weights=val * x[col], minlength=n)
    return rp.astype(np.int32), col.astype(np.int32), val, b, x


# one block, the 64- and 32-thread roundings, both sides of the cluster's limit,
# of 128, 256 and 512 threads on 152 SMs, and the entry point's largest system
SIZES = [(1, 2), (2, 2), (63, 4), (64, 4), (65, 4), (1023, 6), (1025, 6), (6144, 14), (6145, 14), (19456, 6),
         (19457, 6), (38913, 7), (77825, 7), (131072, 6), (131072, 40), (6000, 70)]


@pytest.mark.parametrize("n,couplings", SIZES)
def test_known_solution(built, n, couplings):
    import torch

    from start_gb300 import _native as N

    lib = N.load()
    rp, col, val, b, x = _system(n, couplings, seed=n + couplings)
    dev = [torch.from_numpy(a).cuda() for a in (rp, col, val, b, np.zeros(n))]
    torch.cuda.synchronize()
    runs = []
    for _ in range(2):  # the same twice: the sums' order is fixed
        dev[4].zero_()
        torch.cuda.synchronize()
        it, rr = C.c_int32(), C.c_double()
        rc = lib.spg_pcg_solve_noalloc(n, *[a.data_ptr() for a in dev], RTOL, 500, None, C.byref(it), C.byref(rr))
        assert rc == 0, lib.spg_last_error(None).decode()
        assert rr.value <= RTOL and it.value > 0
        runs.append(dev[4].cpu().numpy())
    assert np.array_equal(runs[0], runs[1])
    assert np.linalg.norm(runs[0] - x) <= 2.0 * RTOL * np.linalg.norm(b)


def test_iteration_cap_keeps_the_iterate(built):
    import torch

    from start_gb300 import _native as N

    lib = N.load()
    rp, col, val, b, x = _system(20000, 6, seed=3)
    dev = [torch.from_numpy(a).cuda() for a in (rp, col, val, b, np.zeros(20000))]
    torch.cuda.synchronize()
    it, rr = C.c_int32(), C.c_double()
    rc = lib.spg_pcg_solve_noalloc(20000, *[a.data_ptr() for a in dev], 1e-14, 3, None, C.byref(it), C.byref(rr))
    assert rc == N.SPG_E_NOT_CONVERGED and it.value == 3 and 0.0 < rr.value < 1.0
    assert np.linalg.norm(dev[4].cpu().numpy() - x) < np.linalg.norm(x)


@pytest.mark.parametrize("cells", [17, 18, 42])
def test_handle_solve_meets_its_residual(built, cells):
    """SELL rows of an unstructured box, cluster and grid forms: the potential's
    own residual b - K phi, in NumPy, within twice the stop tolerance."""
    from start_gb300 import StartPIC, mesh as M
    from start_gb300.workloads import EPS0, _base_params, _zbc

    m = _zbc(M.jitter(M.kuhn_box((cells,) * 3, (0.1,) * 3), 0.2, seed=5))
    eng = StartPIC(m, _base_params(cg_rtol=1e-10))
    rho = np.random.default_rng(cells).uniform(0.0, 1e-7, m.n_nodes)
    phi, it, rr = eng.solve(rho)
    rp, col, val, lift, dual = eng.matrix()
    eng.close()
    b = rho * dual / EPS0 - lift
    b[m.dirichlet_nodes] = m.dirichlet_values
    r = b - np.add.reduceat(val * phi[col], rp[:-1])
    assert it > 10 and rr <= 1e-10
    assert np.linalg.norm(r) <= 2e-10 * np.linalg.norm(b)
