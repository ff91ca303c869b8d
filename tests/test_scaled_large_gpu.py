"""Matrices far from 1 in scale, of orders whose reduction begins with the per-column
kernels (FP64: above 1080). The bars are those of the parity suite, relative to ||H||_2."""
import numpy as np
import pytest

from zquatev_gb300 import _lib, inputs

pytestmark = pytest.mark.gpu

TOL = 1e-12


@pytest.mark.parametrize("scale", [1e-290, 1e-160, 1e-40, 1e40, 1e160, 1e290])
@pytest.mark.parametrize("entry", ["zquatev_fp64_device", "zquatev_device", "zquatev_values_device"])
def test_scale(gpu, entry, scale):
    import torch

    n = 1150
    d0 = torch.from_numpy(np.ascontiguousarray(inputs.random_matrix(n, 8).T)).cuda()
    d, e = d0 * scale, torch.zeros(n, dtype=torch.float64, device="cuda")
    st = torch.cuda.current_stream().cuda_stream
    assert getattr(gpu, entry)(2 * n, d.data_ptr(), 2 * n, e.data_ptr(), st) == 0, _lib.last_error()
    w = e / scale
    a, b = d0[:n, :n].T, d0[:n, n:].T
    h = torch.cat([torch.cat([a, -b.conj()], 1), torch.cat([b, a.conj()], 1)])
    ref = torch.linalg.eigvalsh(h)[::2]
    norm = ref.abs().max()
    assert ((w - ref).abs().max() / norm).item() <= TOL
    if "values" not in entry:
        v = d.T
        assert ((h @ v - v * torch.cat([w, w])).abs().max() / norm).item() <= TOL
        assert (v.mH @ v - torch.eye(2 * n, dtype=v.dtype, device="cuda")).abs().max().item() <= TOL
