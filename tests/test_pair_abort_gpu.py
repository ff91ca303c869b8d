"""A wait of the pair kernel that runs out (residue products): -104, and the next
products are correct. Limits below, about and above one stage's copies, so that the
two CTAs of a pair stop at different stages.

Tolerance: the product's bar elsewhere, 2e-15 of |A| |B| (here k)."""
import pytest

from zquatev_gb300 import _lib

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("limit", [300, 1000, 3000])
@pytest.mark.parametrize("n, k", [(300, 200), (700, 700), (1500, 3000)])
def test_product_recovers(gpu, limit, n, k):
    import torch

    a = torch.ones(k, n, dtype=torch.complex128, device="cuda")
    b = torch.ones(n, k, dtype=torch.complex128, device="cuda")
    c = torch.zeros(n, n, dtype=torch.complex128, device="cuda")
    st = torch.cuda.current_stream().cuda_stream

    def product():
        return gpu.zq_zgemm_accurate(0, 0, n, n, k, a.data_ptr(), n, b.data_ptr(), k, c.data_ptr(), n, st)

    try:
        assert gpu.zq_set_pipeline_wait(limit) == 0
        rc = product()
    finally:
        gpu.zq_set_pipeline_wait(0)
    assert rc == -104 or (rc == 0 and limit > 300), (rc, _lib.last_error())
    assert product() == 0, _lib.last_error()
    assert (c - k).abs().max().item() <= 2e-15 * k
