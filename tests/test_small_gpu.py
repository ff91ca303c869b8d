"""GPU tests of the warp-per-matrix batch solver (zq_small.cu) and of its border with
the path of larger orders: every order of its range (1 to 32; lanes per row and per column change at powers of two), padded leading
dimensions, batches from one matrix to more than the GPU holds at once, matrices at
the ends of the exponent range, uncoupled and degenerate ones.

Tolerance: n - 2 reflectors and about 1.7 n sweeps of rotations per vector, each with
errors of a few eps = 2^-53 that add up like n eps at worst: 64 max(n, 4) eps relative
to ||H|| (2.3e-13 at n = 32), a factor above the growth of either step.
"""
import numpy as np
import pytest

from zquatev_gb300 import _lib, inputs

pytestmark = pytest.mark.gpu

EPS = 2.0 ** -53


def _solve(gpu, mats, pad=0):
    """mats: list of (A, B); returns eigenvalues and vectors of each"""
    import torch

    ns = [len(a) for a, _ in mats]
    lds = [2 * n + (i % 3 if pad else 0) for i, n in enumerate(ns)]
    offs = np.concatenate([[0], np.cumsum([2 * n * ld for n, ld in zip(ns, lds)])]).astype(np.int64)
    eoffs = np.concatenate([[0], np.cumsum(ns)]).astype(np.int64)
    host = np.full(int(offs[-1]), np.nan + 0j)
    for (a, b), n, ld, o in zip(mats, ns, lds, offs):
        blk = np.zeros((ld, 2 * n), np.complex128)
        blk[:n, :n], blk[n:2 * n, :n] = np.tril(a), np.tril(b)  # only the lower triangles are read
        host[o:o + 2 * n * ld] = blk.ravel(order="F")
    d = torch.from_numpy(host).cuda()
    e = torch.zeros(int(eoffs[-1]), dtype=torch.float64, device="cuda")
    n2s, ld2s = np.array([2 * n for n in ns], np.int32), np.array(lds, np.int32)
    rc = gpu.zquatev_batched_device(len(ns), n2s.ctypes.data, ld2s.ctypes.data, offs.ctypes.data, eoffs.ctypes.data,
                                    d.data_ptr(), e.data_ptr(), torch.cuda.current_stream().cuda_stream)
    assert rc == 0, _lib.last_error()
    out, e = d.cpu().numpy(), e.cpu().numpy()
    return [(e[eo:eo + n], out[o:o + 2 * n * ld].reshape(ld, 2 * n, order="F")[:2 * n])
            for n, ld, o, eo in zip(ns, lds, offs, eoffs)]


def _check(mats, results):
    for (a, b), (w, v) in zip(mats, results):
        n = len(a)
        tol = 64 * max(n, 4) * EPS
        norm = max(np.abs(a).max(), np.abs(b).max()) or 1.0
        h = np.block([[a, -b.conj()], [b, a.conj()]]) / norm
        w = w / norm
        ref = np.linalg.eigvalsh(h)[::2]
        hn = max(np.abs(ref).max(), 1.0)
        assert (np.diff(w) >= 0).all()
        assert np.abs(w - ref).max() <= tol * hn
        assert np.linalg.norm(h @ v - v * np.concatenate([w, w]), axis=0).max() <= tol * hn
        assert np.abs(v.conj().T @ v - np.eye(2 * n)).max() <= tol
        assert np.array_equal(v[:n, n:], -v[n:, :n].conj()) and np.array_equal(v[n:, n:], v[:n, :n].conj())


def _random(n, seed):
    d = inputs.random_matrix(n, seed)
    a, b = d[:n, :n], d[n:, :n]
    return (np.tril(a, -1) + np.tril(a, -1).conj().T + np.diag(a.diagonal().real),
            np.tril(b, -1) - np.tril(b, -1).T)


@pytest.mark.parametrize("copies", [1, 40])
def test_every_order(gpu, copies):
    mats = [_random(n, 7 + n) for n in range(1, 33)] * copies
    _check(mats, _solve(gpu, mats, pad=1))


@pytest.mark.parametrize("n", [1, 2, 17, 32])
def test_one_matrix(gpu, n):
    mats = [_random(n, 300 + n)]
    _check(mats, _solve(gpu, mats))


@pytest.mark.parametrize("copies,orders", [(1, (2, 5, 16, 23, 32)), (4, (2, 5, 16, 23, 32)), (1, (33, 40, 75))])
def test_special_matrices(gpu, copies, orders):
    """Few matrices (those from order 16 up take the path of the larger ones), many, and larger ones."""
    mats = []
    for n in orders:
        a, b = _random(n, 500 + n)
        mats += [(a * 1e-290, b * 1e-290), (a * 1e290, b * 1e290)]
        z = np.zeros_like(a)
        mats += [(z, z), (np.eye(n) + 0j, z), (np.diag(np.arange(n) - 2.0) + 0j, z)]
        k = n // 2  # blocks that are uncoupled, or coupled through one tiny entry
        c, f = a.copy(), b.copy()
        c[k:, :k] = c[:k, k:] = f[k:, :k] = f[:k, k:] = 0
        mats.append((c, f))
        c = c.copy()
        c[k, k - 1], c[k - 1, k] = 1e-160j, -1e-160j
        mats.append((c, f))
        u = np.ones((n, 1)) * (1 + 0j)
        mats.append((np.eye(n) + 1e-14 * (u @ u.conj().T), z))
    mats *= copies
    _check(mats, _solve(gpu, mats))


@pytest.mark.parametrize("n", range(1, 11))
def test_single_solve(gpu, n):
    """One matrix per call around the order up to which a warp solves it."""
    import torch

    a, b = _random(n, 800 + n)
    for scale in (1.0, 1e-290, 1e290):
        half = np.zeros((2 * n + 1, 2 * n), np.complex128)
        half[:n, :n], half[n:2 * n, :n] = np.tril(a) * scale, np.tril(b) * scale
        d = torch.from_numpy(np.ascontiguousarray(half.T)).cuda()
        e = torch.full((2 * n,), -3.0, dtype=torch.float64, device="cuda")
        rc = gpu.zquatev_device(2 * n, d.data_ptr(), 2 * n + 1, e.data_ptr(), torch.cuda.current_stream().cuda_stream)
        assert rc == 0, _lib.last_error()
        out, e = d.cpu().numpy().T, e.cpu().numpy()
        assert (e[n:] == -3.0).all() and (out[2 * n] == 0).all()
        _check([(a * scale, b * scale)], [(e[:n], out[:2 * n])])
