"""spg_pcg_solve_noalloc on rows that hold several diagonal entries.

The matrix is the sum of a row's entries. The preconditioner takes the last
diagonal entry that the row stores, and a row whose last one is zero is refused,
whatever the others are. The separate kernels, which serve devices too small for
the one-launch solver, run the same systems (built here with a plan that never
fits): both answer alike.
"""
import ctypes as C
import subprocess

from pathlib import Path

import numpy as np
import pytest

from test_gpu_pcg_resident import RTOL, _system

pytestmark = pytest.mark.gpu

ROOT = Path(__file__).resolve().parent.parent

STUB = r"""
#include <string>
#include "pcg_resident.h"
static std::string message;
namespace spg {
void set_thread_error(const std::string &m) { message = m; }
ResidentPlan resident_plan(int64_t) { return ResidentPlan{}; }
cudaError_t launch_pcg_resident(const ResidentPlan &, ResidentArgs, cudaStream_t) { return cudaErrorNotSupported; }
}
extern "C" const char *spg_last_error(void *) { return message.c_str(); }
"""


@pytest.fixture(scope="module")
def libs(built, tmp_path_factory):
    """The library, and the allocation-free solver alone with its separate kernels."""
    from start_gb300 import _native as N
    from start_gb300.build import ARCH, CSRC, cuda_home

    d = tmp_path_factory.mktemp("noalloc")
    (d / "stub.cu").write_text(STUB)
    so = d / "separate.so"
    subprocess.run([str(cuda_home() / "bin" / "nvcc"), *ARCH, "-O3", "-std=c++17", "-Xcompiler", "-fPIC", "-shared",
                    f"-I{CSRC}", "-o", str(so), str(CSRC / "noalloc.cu"), str(d / "stub.cu")], check=True)
    sep = C.CDLL(str(so))
    sep.spg_last_error.restype = C.c_char_p
    f = N.load().spg_pcg_solve_noalloc
    sep.spg_pcg_solve_noalloc.argtypes, sep.spg_pcg_solve_noalloc.restype = f.argtypes, f.restype
    return {"one launch": N.load(), "separate": sep}


def _solve(lib, rp, ci, av, b, max_iter=500):
    import torch

    n = len(b)
    dev = [torch.from_numpy(np.ascontiguousarray(a)).cuda()
           for a in (np.int32(rp), np.int32(ci), np.float64(av), np.float64(b), np.zeros(n))]
    torch.cuda.synchronize()
    it, rr = C.c_int32(), C.c_double()
    rc = lib.spg_pcg_solve_noalloc(n, *[a.data_ptr() for a in dev], RTOL, max_iter, None, C.byref(it), C.byref(rr))
    return rc, dev[4].cpu().numpy(), it.value, lib.spg_last_error(None).decode()


@pytest.mark.parametrize("which", ["one launch", "separate"])
def test_rows_with_several_diagonal_entries(libs, which):
    from start_gb300 import _native as N

    lib = libs[which]
    rc, x, _, _ = _solve(lib, [0, 2, 3], [0, 0, 1], [1.0, 3.0, 2.0], [8.0, 6.0])
    assert rc == 0 and np.allclose(x, [2.0, 3.0], rtol=1e-10)
    rc, x, _, _ = _solve(lib, [0, 2, 3], [0, 0, 1], [0.0, 4.0, 2.0], [8.0, 6.0])
    assert rc == 0 and np.allclose(x, [2.0, 3.0], rtol=1e-10)
    rc, x, _, msg = _solve(lib, [0, 2, 3], [0, 0, 1], [4.0, 0.0, 2.0], [8.0, 6.0])
    assert rc == N.SPG_E_INVALID and "diagonal" in msg and not x.any()
    rc, x, _, msg = _solve(lib, [0, 3, 4], [0, 0, 0, 1], [5.0, -5.0, 4.0, 2.0], [8.0, 6.0])
    assert rc == 0 and np.allclose(x, [2.0, 3.0], rtol=1e-10)


@pytest.mark.parametrize("n,couplings", [(1, 2), (63, 4), (1025, 6), (6145, 14), (131072, 6)])
def test_separate_kernels_solve_the_known_systems(libs, n, couplings):
    rp, ci, av, b, want = _system(n, couplings, seed=n + couplings)
    its = {}
    for which in libs:
        rc, x, its[which], msg = _solve(libs[which], rp, ci, av, b)
        assert rc == 0, msg
        assert np.linalg.norm(x - want) <= 2.0 * RTOL * np.linalg.norm(b)
    assert abs(its["one launch"] - its["separate"]) <= 1  # the same recurrence, to rounding at the stop test
