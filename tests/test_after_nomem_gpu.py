"""A solve that finds no memory for its workspace (-101, before it touches anything)
leaves the context without one: the next solve of an order solved before makes its own."""
import numpy as np
import pytest

from zquatev_gb300 import _lib, inputs

pytestmark = pytest.mark.gpu

HUGE = 400000  # n2: three buffers of n^2 doubles alone are 960 GB


@pytest.mark.parametrize("entry", ["zquatev_fp64_device", "zquatev_device", "zquatev_values_device"])
@pytest.mark.parametrize("n", [100, 300])
def test_next_solve(gpu, entry, n):
    import torch

    m = inputs.random_matrix(n, n)
    ref = np.linalg.eigvalsh(inputs.full_from_blocks(m[:n, :n], m[n:, :n]))[::2]
    h = torch.from_numpy(np.ascontiguousarray(m.T)).cuda()
    st = torch.cuda.current_stream().cuda_stream
    call = getattr(gpu, entry)
    for _ in range(2):
        d, e = h.clone(), torch.zeros(n, dtype=torch.float64, device="cuda")
        assert call(2 * n, d.data_ptr(), 2 * n, e.data_ptr(), st) == 0, _lib.last_error()
        assert np.abs(e.cpu().numpy() - ref).max() <= 1e-12 * np.abs(ref).max()
        assert call(HUGE, d.data_ptr(), HUGE, e.data_ptr(), st) == -101
