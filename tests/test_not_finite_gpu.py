"""Values that are not numbers stay visible: a matrix or a tridiagonal that holds one gives no
finite eigenvalue and no finite eigenvector, at orders whose merges run on the FP64
pipe and at orders where they run as residue products (600 and up)."""
import numpy as np
import pytest

from zquatev_gb300 import _lib, inputs, solver

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("bad", [float("nan"), float("inf"), float("-inf")], ids=["nan", "inf", "-inf"])
@pytest.mark.parametrize("n", [2, 50, 599, 600, 1300])
@pytest.mark.parametrize("where", ["d", "e"])
def test_tridiagonal(gpu, n, where, bad):
    import torch

    g = torch.Generator(device="cuda").manual_seed(n)
    d = torch.randn(n, dtype=torch.float64, device="cuda", generator=g)
    e = torch.rand(n - 1, dtype=torch.float64, device="cuda", generator=g) + 0.5
    lam, z = torch.zeros(n, dtype=torch.float64, device="cuda"), torch.zeros(n, n, dtype=torch.float64, device="cuda")
    (d if where == "d" else e)[(n - 1) // 2] = bad
    assert solver.stedc_device(d, e, lam, z) == 0, _lib.last_error()
    assert torch.isnan(lam).all()
    assert torch.isnan(z).any(1).all()  # row j of z is eigenvector j
    # and the next solve is not touched by it
    d, e = torch.randn(n, dtype=torch.float64, device="cuda", generator=g), torch.ones(n - 1, dtype=torch.float64, device="cuda")
    assert solver.stedc_device(d, e, lam, z) == 0
    t = torch.diag(d) + torch.diag(e, 1) + torch.diag(e, -1)
    assert (t @ z.T - z.T * lam).abs().max().item() <= 1e-12 * lam.abs().max().item()


@pytest.mark.parametrize("bad", [float("nan"), float("inf")], ids=["nan", "inf"])
@pytest.mark.parametrize("n", [5, 8, 9, 23, 64, 100, 159, 200, 512, 1100])
@pytest.mark.parametrize("entry", ["zquatev_c", "zquatev_fp64_c", "zquatev_values"])
def test_matrix(gpu, entry, n, bad):
    """The drop-in calls: no eigenvalue that looks like one, and the next call is correct."""
    m = inputs.random_matrix(n, n)
    ref = np.linalg.eigvalsh(inputs.full_from_blocks(m[:n, :n], m[n:, :n]))[::2]
    call = getattr(gpu, entry)
    for value in (bad, None):
        d, e = np.array(m, order="F", copy=True), np.zeros(n)
        if value is not None:
            d[n - 1, n // 2] = value
        assert call(2 * n, d.ctypes.data, 2 * n, e.ctypes.data) == 0, _lib.last_error()
        if value is not None:
            assert not np.isfinite(e).any()
    assert np.abs(e - ref).max() <= 1e-12 * np.abs(ref).max()
