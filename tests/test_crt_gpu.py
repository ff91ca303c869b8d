"""GPU tests of the residue-arithmetic products (zq_crt.cu): orders at the edges
of tiles, K stages and exact accumulations, long inner dimensions (the int32
sums are reduced on the way), rows of very different scale, zero rows and
columns, all operand forms; and the divide and conquer whose large merges use
them.

Tolerance of a product: the operands are rounded to 55 bits of their row's
(column's) largest entry, the sums are exact, so the error is below
2 K 2^-56 max|a_i| max|b_j| per part plus the final rounding; with Gaussian
entries (max / rms below 5) that is below 2e-15 |A||B|, the bar of the digit
products.
"""
import numpy as np
import pytest

from zquatev_gb300 import _lib

pytestmark = pytest.mark.gpu


def _op(x, o):
    return {0: x, 1: x.T, 2: x.conj().T, 3: x.conj()}[o]


def _product(gpu, opa, opb, a, b):
    import torch

    m, k = _op(a, opa).shape
    n = _op(b, opb).shape[1]
    da = torch.from_numpy(np.ascontiguousarray(a.T)).cuda()
    db = torch.from_numpy(np.ascontiguousarray(b.T)).cuda()
    dc = torch.full((n, m + 3), 7.0, dtype=torch.complex128, device="cuda")
    rc = gpu.zq_zgemm_accurate(opa, opb, m, n, k, da.data_ptr(), a.shape[0], db.data_ptr(), b.shape[0], dc.data_ptr(),
                               m + 3, torch.cuda.current_stream().cuda_stream)
    torch.cuda.synchronize()
    assert rc == 0, _lib.last_error()
    assert (dc[:, m:] == 7.0).all()
    return dc[:, :m].cpu().numpy().T


def _gauss(rng, shape):
    return rng.standard_normal(shape) + 1j * rng.standard_normal(shape)


@pytest.mark.parametrize("m,n,k", [(1, 1, 1), (3, 5, 63), (31, 33, 64), (255, 17, 65), (256, 256, 127), (257, 255, 128),
                                   (40, 300, 511), (64, 513, 512), (100, 70, 513), (8, 9, 40000)])
@pytest.mark.parametrize("opa,opb", [(0, 0), (1, 3), (2, 1), (3, 2)])
def test_product_orders(gpu, m, n, k, opa, opb):
    rng = np.random.default_rng(m + 7 * n + 13 * k + opa)
    a = _gauss(rng, (k, m) if opa in (1, 2) else (m, k))
    b = _gauss(rng, (n, k) if opb in (1, 2) else (k, n))
    c = _product(gpu, opa, opb, a, b)
    exact = _op(a, opa).astype(np.clongdouble) @ _op(b, opb).astype(np.clongdouble)
    scale = np.abs(_op(a, opa)) @ np.abs(_op(b, opb))
    tol = 2e-15 if k > 1 else 2.0 ** -50  # one term: no averaging over the row
    assert (np.abs(c - exact.astype(np.complex128)) / scale).max() < tol


def test_product_scales_and_zeros(gpu):
    rng = np.random.default_rng(3)
    a, b = _gauss(rng, (70, 90)), _gauss(rng, (90, 60))
    a *= 10.0 ** rng.integers(-140, 140, 70)[:, None]
    b *= 10.0 ** rng.integers(-140, 140, 60)[None, :]
    a[5] = 0
    b[:, 7] = 0
    a[9, 1:] = 0
    c = _product(gpu, 0, 0, a, b)
    exact = (a.astype(np.clongdouble) @ b.astype(np.clongdouble)).astype(np.complex128)
    assert (c[5] == 0).all() and (c[:, 7] == 0).all()
    rows = np.abs(a).max(1)[:, None] * np.abs(b).max(0)[None, :]
    live = rows > 0
    assert (np.abs(c - exact)[live] / rows[live]).max() < 90 * 2.0 ** -53


@pytest.mark.parametrize("n", [599, 600, 601, 777, 1201])
def test_divide_and_conquer_merges(gpu, n):
    import torch
    from zquatev_gb300 import solver

    g = torch.Generator(device="cuda").manual_seed(n)
    d = torch.randn(n, dtype=torch.float64, device="cuda", generator=g)
    e = torch.rand(n - 1, dtype=torch.float64, device="cuda", generator=g) + 0.1
    lam, z = torch.empty_like(d), torch.empty(n, n, dtype=torch.float64, device="cuda")
    assert solver.stedc_device(d, e, lam, z) == 0
    torch.cuda.synchronize()
    t = torch.diag(d) + torch.diag(e, 1) + torch.diag(e, -1)
    norm = t.abs().sum(0).max()
    v = z.T
    assert ((t @ v - v * lam).abs().max() / norm).item() < 1e-14
    assert (v.T @ v - torch.eye(n, dtype=torch.float64, device="cuda")).abs().max().item() < 1e-13
    assert ((torch.linalg.eigvalsh(t) - lam).abs().max() / norm).item() < 1e-14
