"""The first re-sort of a mixed-form set takes no device memory of its own: its
records (32 bytes a particle) lie in the walk queue's. Another program on the GPU
could allocate meanwhile, so the bar is half of the records' size."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_first_sort_of_a_mixed_set_allocates_no_records(built):
    import torch

    from start_gb300 import StartPIC, mesh as M
    from start_gb300.workloads import _base_params, _zbc

    n = 4_000_000
    m = _zbc(M.kuhn_box((12, 12, 12), (0.1,) * 3))
    rng = np.random.default_rng(1)
    with StartPIC(m, _base_params(precision=1)) as e:
        e.set_particles(rng.uniform(0.001, 0.099, (n, 3)), np.zeros((n, 3)))
        before = e.particles()
        free = torch.cuda.mem_get_info()[0]
        e.resort()
        assert free - torch.cuda.mem_get_info()[0] < 16 * n
        after = e.particles()
    for k in ("pos", "vel", "tet", "flags"):
        assert np.array_equal(before[k], after[k])
