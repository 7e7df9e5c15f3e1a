"""The one-launch Jacobi PCG with one exchange of sums per iteration: at the edges of
its launch shapes, and against textbook CG in NumPy step by step.

With the stop at max_iter = k the returned x is CG's k-th iterate. Both run the
same recurrences in FP64; the difference after k <= 12 steps of a system with
condition below 20 is a few hundred eps of ||x||, 1e-12 is the bound. A diagonal
system ends after one step whatever its size.
"""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _system(n, seed):
    """Symmetric, a_ii = 1 + 1.5 sum |a_ij|: spectrum of D^-1 A within [1/3, 5/3]."""
    rng = np.random.default_rng(seed)
    i, j = rng.integers(0, n, 3 * n), rng.integers(0, n, 3 * n)
    key = np.unique((np.minimum(i, j) * n + np.maximum(i, j))[i != j])
    i, j = key // n, key % n
    v = rng.uniform(-1.0, 1.0, len(i))
    diag = np.full(n, 1.0)
    np.add.at(diag, i, 1.5 * np.abs(v))
    np.add.at(diag, j, 1.5 * np.abs(v))
    row, col = np.concatenate([i, j, np.arange(n)]), np.concatenate([j, i, np.arange(n)])
    val = np.concatenate([v, v, diag])
    o = np.lexsort((col, row))
    row, col, val = row[o], col[o], val[o]
    rp = np.concatenate([[0], np.cumsum(np.bincount(row, minlength=n))]).astype(np.int32)
    return rp, row, col.astype(np.int32), val, diag, rng.normal(size=n)


def _solve(rp, col, val, b, rtol, max_iter):
    import torch

    from start_gb300 import _native as N

    lib = N.load()
    dev = [torch.from_numpy(a).cuda() for a in (rp, col, val, b, np.zeros(len(b)))]
    torch.cuda.synchronize()
    it, rr = C.c_int32(), C.c_double()
    rc = lib.spg_pcg_solve_noalloc(len(b), *[a.data_ptr() for a in dev], rtol, max_iter, None, C.byref(it), C.byref(rr))
    return rc, it.value, rr.value, dev[4].cpu().numpy()


# threads per block 64, 96, 128 (a cluster and both sides of its limit), 256, 512, 1024
@pytest.mark.parametrize("n", [1, 2, 900, 1500, 4096, 4097, 19457, 38913, 77825])
def test_iterates_are_those_of_cg(built, n):
    rp, row, col, val, diag, b = _system(n, n)
    mul = lambda p: np.bincount(row, weights=val * p[col], minlength=n)
    x, r = np.zeros(n), b.copy()
    z = r / diag
    p, rz = z.copy(), float(r @ (r / diag))
    want = []
    for _ in range(12):
        q = mul(p)
        a = rz / (p @ q)
        x = x + a * p
        r = r - a * q
        want.append((x, np.linalg.norm(r) / np.linalg.norm(b)))
        z = r / diag
        new = float(r @ z)
        p, rz = z + (new / rz) * p, new
        if want[-1][1] < 1e-9:
            break
    for k in {1, 2, len(want)} - {0}:
        if k > len(want):
            continue
        rc, it, rr, got = _solve(rp, col, val, b, 1e-14, k)
        assert it == k and rc in (0, -4)
        assert np.linalg.norm(got - want[k - 1][0]) <= 1e-12 * np.linalg.norm(want[k - 1][0])
        assert abs(rr - want[k - 1][1]) <= 1e-10 * max(want[k - 1][1], 1e-3)


@pytest.mark.parametrize("n", [5, 3000, 6000])
def test_diagonal_system_takes_one_step(built, n):
    rng = np.random.default_rng(n)
    d = rng.uniform(0.5, 2.0, n)
    b = rng.normal(size=n)
    rc, it, rr, x = _solve(np.arange(n + 1, dtype=np.int32), np.arange(n, dtype=np.int32), d, b, 1e-12, 50)
    assert rc == 0 and it == 1 and rr <= 1e-12
    assert np.allclose(x, b / d, rtol=1e-13, atol=0)
