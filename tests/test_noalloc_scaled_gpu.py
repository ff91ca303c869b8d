"""zquatev_device_noalloc on matrices far from 1 in scale, and with a value that is not a
number (info above 0, as from every kernel with an implicit QL)."""
import numpy as np
import pytest

from zquatev_gb300 import _lib, inputs

pytestmark = pytest.mark.gpu

TOL = 1e-12


@pytest.mark.parametrize("scale", [1e-290, 1e-160, 1e-40, 1.0, 1e40, 1e160, 1e290])
@pytest.mark.parametrize("n", [2, 37, 200])
def test_scale(gpu, n, scale):
    import torch

    d0 = torch.from_numpy(np.ascontiguousarray(inputs.random_matrix(n, 8).T)).cuda()
    d, e = d0 * scale, torch.zeros(n, dtype=torch.float64, device="cuda")
    rc = gpu.zquatev_device_noalloc(2 * n, d.data_ptr(), 2 * n, e.data_ptr(), torch.cuda.current_stream().cuda_stream)
    assert rc == 0, _lib.last_error()
    w, v = e / scale, d.T
    a, b = d0[:n, :n].T, d0[:n, n:].T
    h = torch.cat([torch.cat([a, -b.conj()], 1), torch.cat([b, a.conj()], 1)])
    norm = w.abs().max()
    assert ((h @ v - v * torch.cat([w, w])).abs().max() / norm).item() <= TOL
    assert (v.mH @ v - torch.eye(2 * n, dtype=v.dtype, device="cuda")).abs().max().item() <= TOL


@pytest.mark.parametrize("n", [5, 60])
def test_not_a_number(gpu, n):
    import torch

    d = torch.from_numpy(np.ascontiguousarray(inputs.random_matrix(n, 8).T)).cuda()
    d[1, 1] = float("nan")
    e = torch.zeros(n, dtype=torch.float64, device="cuda")
    rc = gpu.zquatev_device_noalloc(2 * n, d.data_ptr(), 2 * n, e.data_ptr(), torch.cuda.current_stream().cuda_stream)
    assert rc > 0
    assert not torch.isfinite(e).all()
