"""Batches at the limits of a launch and of the memory."""
import numpy as np
import pytest

from zquatev_gb300 import _lib, inputs, solver

pytestmark = pytest.mark.gpu


def _copies(n, count, seed=3):
    """`count` copies of one matrix, with what zquatev_batched_device takes."""
    import torch

    n2 = np.full(count, 2 * n, np.int32)
    offs = np.arange(count, dtype=np.int64) * (4 * n * n)
    eoffs = np.arange(count, dtype=np.int64) * n
    one = torch.from_numpy(np.ascontiguousarray(inputs.random_matrix(n, seed).T)).cuda()
    d = one[None].repeat(count, 1, 1)
    return d, torch.zeros(count, n, dtype=torch.float64, device="cuda"), (n2, n2.copy(), offs, eoffs)


def _run(gpu, d, e, args):
    import torch

    return gpu.zquatev_batched_device(len(args[0]), *(a.ctypes.data for a in args), d.data_ptr(), e.data_ptr(),
                                      torch.cuda.current_stream().cuda_stream)


def _check(n, d, e, seed=3):
    import torch

    m = inputs.random_matrix(n, seed)
    h = torch.from_numpy(inputs.full_from_blocks(m[:n, :n], m[n:, :n])).cuda()
    v, w = d[0].T, e[0]
    norm = w.abs().max()
    assert ((h @ v - v * torch.cat([w, w])).abs().max() / norm).item() <= 1e-12
    assert (v.mH @ v - torch.eye(2 * n, dtype=v.dtype, device="cuda")).abs().max().item() <= 1e-12
    assert (e == e[0]).all() and (d == d[0]).all()


def test_more_matrices_than_a_grid_dimension(gpu):
    d, e, args = _copies(33, 65537)
    assert _run(gpu, d, e, args) == 0, _lib.last_error()
    _check(33, d, e)
