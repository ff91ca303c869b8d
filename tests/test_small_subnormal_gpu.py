"""Matrices whose entries are all subnormal numbers, at the orders a warp solves: small
integers times 2^-1070, so that nothing is lost on the way in.

Tolerance: an eigenvalue is stored in units of 2^-1074, a sixteenth of the unit
here, so it may be a thirty-second off; the eigenvectors keep the bars of the other tests."""
import numpy as np
import pytest

from zquatev_gb300 import _lib

pytestmark = pytest.mark.gpu

UNIT = 2.0 ** -1070


def _integers(n, seed):
    r = np.random.default_rng(seed)
    x = r.integers(-8, 9, (n, n)) + 1j * r.integers(-8, 9, (n, n))
    y = r.integers(-8, 9, (n, n)) + 1j * r.integers(-8, 9, (n, n))
    return np.triu(x, 1) + np.triu(x, 1).conj().T + np.diag(x.real.diagonal()), np.triu(y, 1) - np.triu(y, 1).T


def _check(n, a, b, v, w):
    h = np.block([[a, -b.conj()], [b, a.conj()]])
    ref = np.linalg.eigvalsh(h)[::2]
    norm = np.abs(ref).max()
    got = w * 2.0 ** 1000 * 2.0 ** 70
    assert np.abs(got - ref).max() <= 1 / 32 + 1e-12 * norm
    lam = np.concatenate([ref, ref])
    assert np.abs(h @ v - v * lam).max() <= 1e-12 * norm
    assert np.abs(v.conj().T @ v - np.eye(2 * n)).max() <= 1e-12


@pytest.mark.parametrize("n", [2, 3, 8])
def test_single(gpu, n):
    a, b = _integers(n, n)
    d = np.zeros((2 * n, 2 * n), dtype=np.complex128, order="F")
    d[:n, :n], d[n:, :n] = a * UNIT, b * UNIT
    e = np.zeros(n)
    assert gpu.zquatev_c(2 * n, d.ctypes.data, 2 * n, e.ctypes.data) == 0, _lib.last_error()
    _check(n, a, b, d, e)


@pytest.mark.parametrize("n", [3, 19, 32])
def test_batch(gpu, n):
    import torch

    count = 200
    a, b = _integers(n, 50 + n)
    d = np.zeros((2 * n, 2 * n), dtype=np.complex128, order="F")
    d[:n, :n], d[n:, :n] = a * UNIT, b * UNIT
    n2 = np.full(count, 2 * n, np.int32)
    offs = np.arange(count, dtype=np.int64) * (4 * n * n)
    eoffs = np.arange(count, dtype=np.int64) * n
    dd = torch.from_numpy(np.ascontiguousarray(d.T)).cuda()[None].repeat(count, 1, 1)
    de = torch.zeros(count, n, dtype=torch.float64, device="cuda")
    assert gpu.zquatev_batched_device(count, n2.ctypes.data, n2.ctypes.data, offs.ctypes.data, eoffs.ctypes.data,
                                      dd.data_ptr(), de.data_ptr(), 0) == 0, _lib.last_error()
    for i in (0, count - 1):
        _check(n, a, b, dd[i].cpu().numpy().T, de[i].cpu().numpy())


def test_zero_matrix(gpu):
    d, e = np.zeros((12, 12), dtype=np.complex128, order="F"), np.ones(6)
    assert gpu.zquatev_c(12, d.ctypes.data, 12, e.ctypes.data) == 0
    assert (e == 0).all() and np.abs(d.conj().T @ d - np.eye(12)).max() <= 1e-15
