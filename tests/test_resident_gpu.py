"""GPU tests of the shared-memory resident reduction (zq_resident.cu) and the
direct back-transform (zq_applyq.cu): orders at the edges of tiles, of row
passes, of the cluster, group and direct-application ranges, and where the
last columns of a larger matrix are handed over.

Tolerance: the bars of the parity suite (residual, orthonormality and
eigenvalue error 1e-12 relative to ||H||_2), which leave a factor of ~200 over
n eps for the largest order here.
"""
import numpy as np
import pytest

from zquatev_gb300 import _lib, inputs

pytestmark = pytest.mark.gpu

TOL = 1e-12


def _solve(gpu, n, path, scale=1.0, pad=0, seed=5):
    import torch

    d0 = torch.from_numpy(np.ascontiguousarray(inputs.random_matrix(n, seed + n).T)).cuda() * scale
    d = torch.zeros(2 * n, 2 * n + pad, dtype=torch.complex128, device="cuda")
    d[:, : 2 * n] = d0
    e = torch.zeros(2 * n, dtype=torch.float64, device="cuda")
    st = torch.cuda.current_stream().cuda_stream
    if path == "fp64":
        rc = gpu.zquatev_fp64_device(2 * n, d.data_ptr(), 2 * n + pad, e.data_ptr(), st)
    else:
        rc = gpu.zquatev_refined_device(2 * n, d.data_ptr(), 2 * n + pad, e.data_ptr(), st, 1)
    torch.cuda.synchronize()
    assert rc == 0, _lib.last_error()
    h, v, w = d0.T, d[:, : 2 * n].T, e[:n]
    ref = torch.linalg.eigvalsh(h)[::2]
    norm = ref.abs().max()
    assert ((w - ref).abs().max() / norm).item() <= TOL
    assert ((h @ v - v * torch.cat([w, w])).abs().max() / norm).item() <= TOL
    assert (v.mH @ v - torch.eye(2 * n, device="cuda", dtype=v.dtype)).abs().max().item() <= TOL
    assert torch.equal(v[:n, n:], -v[n:, :n].conj()) and torch.equal(v[n:, n:], v[:n, :n].conj())


@pytest.mark.parametrize("n", [1, 2, 3, 4, 7, 8, 9, 15, 16, 17, 31, 32, 33, 63, 64, 65, 96, 97, 128, 129, 193, 257, 321,
                               385, 449, 513, 641, 800, 801, 1080, 1081, 1100])
def test_fp64_orders(gpu, n):
    _solve(gpu, n, "fp64")


@pytest.mark.parametrize("n", [48, 49, 127, 128, 447, 448, 449, 609, 1023, 1663, 1664, 1665, 1690])
def test_refined_orders(gpu, n):
    _solve(gpu, n, "refined")


@pytest.mark.parametrize("scale", [1e-140, 1e-30, 1e30, 1e140])
def test_fp64_scaled_input(gpu, scale):
    _solve(gpu, 70, "fp64", scale=scale, pad=3)


def test_fp64_structured_columns(gpu):
    """Columns that are already reduced, zero columns and a zero leading entry."""
    import torch

    n = 40
    a = np.zeros((n, n), dtype=np.complex128)
    b = np.zeros((n, n), dtype=np.complex128)
    a[np.arange(n), np.arange(n)] = np.linspace(-1, 1, n)
    a[5, 3], a[3, 5] = 0.5j, -0.5j          # x_1 = 0 below column 3
    b[20, 18], b[18, 20] = 0.25, -0.25      # the B part only
    a[30, 29] = a[29, 30] = 0.1             # already subdiagonal
    d0 = torch.from_numpy(np.ascontiguousarray(inputs.pack_left_half(a, b).T)).cuda()
    d, e = d0.clone(), torch.zeros(2 * n, dtype=torch.float64, device="cuda")
    st = torch.cuda.current_stream().cuda_stream
    assert gpu.zquatev_fp64_device(2 * n, d.data_ptr(), 2 * n, e.data_ptr(), st) == 0
    torch.cuda.synchronize()
    h, v, w = d0.T, d.T, e[:n]
    assert (w - torch.linalg.eigvalsh(h)[::2]).abs().max().item() <= TOL
    assert (h @ v - v * torch.cat([w, w])).abs().max().item() <= TOL
    assert (v.mH @ v - torch.eye(2 * n, device="cuda", dtype=v.dtype)).abs().max().item() <= TOL


@pytest.mark.parametrize("path", ["fp64", "refined"])
@pytest.mark.parametrize("tiny", [1e-8, 1e-14, 1e-20, 1e-78, 1e-100, 1e-160])
def test_weakly_coupled_blocks(gpu, path, tiny):
    """Two blocks joined by entries far below the matrix's size: the columns at
    the seam shrink to the coupling, and their reflectors must stay unitary."""
    import torch

    n = 90
    a, b = inputs.random_blocks(n, 77)
    a[:30, 30:] *= tiny
    a[30:, :30] *= tiny
    b[:30, 30:] *= tiny
    b[30:, :30] *= tiny
    d0 = torch.from_numpy(np.ascontiguousarray(inputs.pack_left_half(a, b).T)).cuda()
    d, e = d0.clone(), torch.zeros(2 * n, dtype=torch.float64, device="cuda")
    st = torch.cuda.current_stream().cuda_stream
    if path == "fp64":
        rc = gpu.zquatev_fp64_device(2 * n, d.data_ptr(), 2 * n, e.data_ptr(), st)
    else:
        rc = gpu.zquatev_refined_device(2 * n, d.data_ptr(), 2 * n, e.data_ptr(), st, 1)
    torch.cuda.synchronize()
    assert rc == 0, _lib.last_error()
    h, v, w = d0.T, d.T, e[:n]
    norm = w.abs().max()
    assert ((w - torch.linalg.eigvalsh(h)[::2]).abs().max() / norm).item() <= TOL
    assert ((h @ v - v * torch.cat([w, w])).abs().max() / norm).item() <= TOL
    assert (v.mH @ v - torch.eye(2 * n, device="cuda", dtype=v.dtype)).abs().max().item() <= TOL
