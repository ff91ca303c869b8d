"""zq_release_workspace gives back what the solves keep."""
import gc

import numpy as np
import pytest

from zquatev_gb300 import _lib, inputs

pytestmark = pytest.mark.gpu

MB = 1 << 20


def _free():
    import torch

    gc.collect()
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    return torch.cuda.mem_get_info()[0]


def _held(gpu):
    """What zq_release_workspace gives back now."""
    before = _free()
    assert gpu.zq_release_workspace() == 0
    return _free() - before


@pytest.mark.parametrize("entry", ["zquatev_device", "zquatev_values_device"])
def test_solve(gpu, entry):
    """n = 1000: the refinement's buffers alone are ten n x n complex arrays and the products' residues, 500 MB."""
    import torch

    n = 1000
    d = torch.from_numpy(np.ascontiguousarray(inputs.random_matrix(n, 1).T)).cuda()
    e = torch.zeros(n, dtype=torch.float64, device="cuda")
    rc = getattr(gpu, entry)(2 * n, d.data_ptr(), 2 * n, e.data_ptr(), torch.cuda.current_stream().cuda_stream)
    assert rc == 0, _lib.last_error()
    assert _held(gpu) >= 500 * MB
    assert _held(gpu) <= 2 * MB


def test_batch(gpu):
    """Matrices of a warp each: the CTA kernel's workspace, 0.5 MB for each of 304 CTAs, is kept."""
    import torch

    n, count = 20, 1000
    n2 = np.full(count, 2 * n, np.int32)
    offs = np.arange(count, dtype=np.int64) * (4 * n * n)
    eoffs = np.arange(count, dtype=np.int64) * n
    d = torch.from_numpy(np.ascontiguousarray(inputs.random_matrix(n, 1).T)).cuda()[None].repeat(count, 1, 1)
    e = torch.zeros(count * n, dtype=torch.float64, device="cuda")
    rc = gpu.zquatev_batched_device(count, n2.ctypes.data, n2.ctypes.data, offs.ctypes.data, eoffs.ctypes.data,
                                    d.data_ptr(), e.data_ptr(), torch.cuda.current_stream().cuda_stream)
    assert rc == 0, _lib.last_error()
    assert _held(gpu) >= 120 * MB


def test_product(gpu):
    """Released right after the call, while its scratch is not yet free in stream order: 1 GB at N = 2048."""
    import torch

    n = 2048
    a = torch.ones(n, n, dtype=torch.complex128, device="cuda")
    c = torch.zeros_like(a)
    st = torch.cuda.current_stream().cuda_stream
    for _ in range(2):
        assert gpu.zq_zgemm_accurate(0, 0, n, n, n, a.data_ptr(), n, a.data_ptr(), n, c.data_ptr(), n, st) == 0
        before = _free()
        assert gpu.zq_zgemm_accurate(0, 0, n, n, n, a.data_ptr(), n, a.data_ptr(), n, c.data_ptr(), n, st) == 0
        torch.cuda._sleep(1000000)
        assert gpu.zq_release_workspace() == 0
        assert _free() - before >= 500 * MB


def test_solves_go_on_after_it(gpu):
    import torch

    st = torch.cuda.current_stream().cuda_stream
    for n in (30, 300, 30):
        m = inputs.random_matrix(n, n)
        ref = np.linalg.eigvalsh(inputs.full_from_blocks(m[:n, :n], m[n:, :n]))[::2]
        d, e = torch.from_numpy(np.ascontiguousarray(m.T)).cuda(), torch.zeros(n, dtype=torch.float64, device="cuda")
        assert gpu.zquatev_device(2 * n, d.data_ptr(), 2 * n, e.data_ptr(), st) == 0
        assert np.abs(e.cpu().numpy() - ref).max() <= 1e-12 * np.abs(ref).max()
        assert gpu.zq_release_workspace() == 0
