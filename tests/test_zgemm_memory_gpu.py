"""zq_zgemm_accurate at the limits of its residues: where their scratch (240 N^2 bytes)
does not fit beside the operands but the digit slices' (96 N^2) does, and where the
inner dimension is longer than their grid."""
import gc

import pytest

from zquatev_gb300 import _lib

pytestmark = pytest.mark.gpu


def test_product_without_room_for_residues(gpu):
    import torch

    n = 4096
    g = torch.Generator(device="cuda").manual_seed(1)
    a = torch.randn(n, n, dtype=torch.complex128, device="cuda", generator=g)
    b = torch.randn(n, n, dtype=torch.complex128, device="cuda", generator=g)
    c = torch.zeros_like(a)
    st = torch.cuda.current_stream().cuda_stream
    ref = (b[:8] @ a).clone()          # column-major: C = A B is (b @ a) here
    assert gpu.zq_zgemm_accurate(0, 0, n, n, n, a.data_ptr(), n, b.data_ptr(), n, c.data_ptr(), n, st) == 0
    full = c.clone()
    torch.cuda.synchronize()           # (what is not yet free in stream order stays in the pool)
    gpu.zq_release_workspace()
    gc.collect()
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    ballast = torch.empty(torch.cuda.mem_get_info()[0] - (5 << 29), dtype=torch.uint8, device="cuda")  # 2.5 GB left
    try:
        c.zero_()
        rc = gpu.zq_zgemm_accurate(0, 0, n, n, n, a.data_ptr(), n, b.data_ptr(), n, c.data_ptr(), n, st)
        torch.cuda.synchronize()
        gpu.zq_release_workspace()
    finally:
        del ballast
        gc.collect()
        torch.cuda.empty_cache()
    assert rc == 0, _lib.last_error()
    scale = (a.abs().max() * b.abs().max() * n).item()
    assert (c[:8] - ref).abs().max().item() <= 1e-14 * scale
    assert (c - full).abs().max().item() <= 1e-14 * scale


def test_long_inner_dimension(gpu):
    """65535 blocks of 64 terms and a few more (A^T B: both contiguous along the terms)."""
    import torch

    k = 64 * 65535 + 70
    g = torch.Generator(device="cuda").manual_seed(2)
    a = torch.randn(2, k, dtype=torch.complex128, device="cuda", generator=g)   # k x 2, column-major
    b = torch.randn(2, k, dtype=torch.complex128, device="cuda", generator=g)
    c = torch.zeros(2, 2, dtype=torch.complex128, device="cuda")
    rc = gpu.zq_zgemm_accurate(1, 0, 2, 2, k, a.data_ptr(), k, b.data_ptr(), k, c.data_ptr(), 2,
                               torch.cuda.current_stream().cuda_stream)
    assert rc == 0, _lib.last_error()
    bound = b.abs() @ a.abs().T
    assert ((c - b @ a.T).abs() / bound).max().item() <= 1e-13
    torch.cuda.synchronize()
    gpu.zq_release_workspace()
