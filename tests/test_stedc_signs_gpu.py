"""zq_stedc_device takes off-diagonal entries of either sign."""
import pytest

from zquatev_gb300 import _lib, solver

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [2, 3, 33, 64, 65, 700, 1025, 2500])
@pytest.mark.parametrize("kind", ["toeplitz", "random"])
@pytest.mark.parametrize("pad", [0, 3])
def test_signs(gpu, n, kind, pad):
    import torch

    g = torch.Generator(device="cuda").manual_seed(n)
    if kind == "toeplitz":
        d = torch.full((n,), 2.0, dtype=torch.float64, device="cuda")
        e = torch.full((n - 1,), -1.0, dtype=torch.float64, device="cuda")
    else:
        d = torch.randn(n, dtype=torch.float64, device="cuda", generator=g)
        e = torch.randn(n - 1, dtype=torch.float64, device="cuda", generator=g)
        e[n // 3] = 0.0
    e0 = e.clone()
    lam = torch.zeros(n, dtype=torch.float64, device="cuda")
    buf = torch.full((n, n + pad), 7.0, dtype=torch.float64, device="cuda")
    rc = gpu.zq_stedc_device(n, d.data_ptr(), e.data_ptr(), lam.data_ptr(), buf.data_ptr(), n + pad,
                             torch.cuda.current_stream().cuda_stream)
    assert rc == 0, _lib.last_error()
    z = buf[:, :n].T
    t = torch.diag(d) + torch.diag(e, 1) + torch.diag(e, -1)
    norm = lam.abs().max().item()
    assert (t @ z - z * lam).abs().max().item() <= 1e-13 * norm
    assert (z.T @ z - torch.eye(n, dtype=z.dtype, device="cuda")).abs().max().item() <= 1e-13
    assert (lam.diff() >= 0).all() and torch.equal(e, e0) and (buf[:, n:] == 7.0).all()
