"""GPU test of the FP32 trailing update (zq_tridiag.cu) through the refined path: orders
above what the resident reduction holds, odd and even, panels narrower and wider than
the update's chunk of 16 reflectors and not a multiple of it.

Tolerance: the parity suite's 1e-12, and the FP32 start must let the refinement
converge by itself.
"""
import numpy as np
import pytest

from zquatev_gb300 import inputs, solver

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,nb", [(1701, 16), (1730, 7), (1792, 40), (1669, 128)])
def test_panels(gpu, n, nb):
    import torch

    half = torch.from_numpy(np.ascontiguousarray(inputs.random_matrix(n, n).T)).cuda()
    d, eig = half.clone(), torch.zeros(2 * n, dtype=torch.float64, device="cuda")
    keep = gpu.zq_get_block_size()
    try:
        assert gpu.zq_set_block_size(nb) == 0
        assert gpu.zquatev_refined_device(2 * n, d.data_ptr(), 2 * n, eig.data_ptr(),
                                          torch.cuda.current_stream().cuda_stream, 1) == 0
    finally:
        assert gpu.zq_set_block_size(keep) == 0
    assert not solver.refine_stats()[2]
    a, b, w, v = half.T[:n, :n], half.T[n:, :n], eig[:n], d.T[:, :n]
    # the left half's residual: H v = lambda v, v = [u; x], H = (A -B*; B A*)
    top = a @ v[:n] - b.conj() @ v[n:] - v[:n] * w
    bottom = b @ v[:n] + a.conj() @ v[n:] - v[n:] * w
    assert max(top.abs().max().item(), bottom.abs().max().item()) <= 1e-12 * w.abs().max().item()
    assert (v.mH @ v - torch.eye(n, dtype=v.dtype, device="cuda")).abs().max().item() <= 1e-12
