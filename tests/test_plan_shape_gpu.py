"""A plan with a fixed launch shape solves small orders as an unplanned batch does: a
warp each up to the default switch size (the same kernel, hence the same bits)."""
import numpy as np
import pytest

from zquatev_gb300 import _lib, inputs, solver

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ctas_per_sm", [1, 2, 4])
@pytest.mark.parametrize("n", [3, 19, 32])
def test_fixed_shape_takes_the_warp_kernel(gpu, n, ctas_per_sm):
    import torch

    count = 200
    n2 = np.full(count, 2 * n, np.int32)
    offs = np.arange(count, dtype=np.int64) * (4 * n * n)
    eoffs = np.arange(count, dtype=np.int64) * n
    args = (n2, n2.copy(), offs, eoffs)
    d0 = torch.stack([torch.from_numpy(np.ascontiguousarray(inputs.random_matrix(n, i).T)) for i in range(count)]).cuda()
    d1, e1 = d0.clone(), torch.zeros(count, n, dtype=torch.float64, device="cuda")
    assert gpu.zquatev_batched_device(count, *(a.ctypes.data for a in args), d1.data_ptr(), e1.data_ptr(), 0) == 0, \
        _lib.last_error()
    plan = solver.BatchPlan(*args, ctas_per_sm=ctas_per_sm)
    d2, e2 = d0.clone(), torch.zeros_like(e1)
    plan.run(d2, e2)
    assert plan.info() == 0 and plan.shape()["warp_max_n"] == 32
    plan.close()
    assert torch.equal(d1, d2) and torch.equal(e1, e2)
