"""GPU tests of the eigenvalues-only calls around the order from which they take the
refined path: against the eigenvalues of the FP64 path, on matrices whose refinement
does not converge by itself, on the host entry, and under stream capture, where the
call stays on the FP64 path.

Tolerance: both paths carry errors of a few eps per step of a backward stable
reduction: 1e-12 relative to ||H||, the bar of the parity suite.
"""
import numpy as np
import pytest

from zquatev_gb300 import _lib, inputs, solver

pytestmark = pytest.mark.gpu

TOL = 1e-12


def _values(gpu, half, n, path=None):
    import torch

    if path is not None:
        gpu.zq_set_path(path)
    try:
        d = torch.from_numpy(np.ascontiguousarray(half.T)).cuda()
        e = torch.zeros(2 * n, dtype=torch.float64, device="cuda")
        _lib.check(gpu.zquatev_values_device(2 * n, d.data_ptr(), 2 * n, e.data_ptr(),
                                             torch.cuda.current_stream().cuda_stream), "values")
        return e[:n].cpu().numpy()
    finally:
        gpu.zq_set_path(2)


@pytest.mark.parametrize("n", [219, 220, 221, 383, 900])
def test_paths_agree(gpu, n):
    half = inputs.random_matrix(n, n)
    auto, fp64 = _values(gpu, half, n), _values(gpu, half, n, 0)
    assert (np.diff(auto) >= 0).all()
    assert np.abs(auto - fp64).max() <= TOL * np.abs(fp64).max()
    if n < 220:
        assert np.array_equal(auto, fp64)
    eig = np.zeros(2 * n)
    work = np.array(half, order="F", copy=True)
    _lib.check(gpu.zquatev_values(2 * n, work.ctypes.data, 2 * n, eig.ctypes.data), "values")
    assert np.array_equal(eig[:n], auto)


def test_degenerate(gpu):
    n = 400
    a = np.diag(np.repeat(np.arange(4.0), n // 4)).astype(np.complex128)
    u, _ = np.linalg.qr(np.random.default_rng(5).standard_normal((n, n)))
    half = np.zeros((2 * n, 2 * n), np.complex128, order="F")
    half[:n, :n] = u @ a @ u.T
    half[:n, :n] = (half[:n, :n] + half[:n, :n].T) / 2
    w = _values(gpu, half, n)
    assert np.abs(w - np.repeat(np.arange(4.0), n // 4)).max() <= TOL * 3


def test_under_capture(gpu):
    import torch

    n = 400
    half = inputs.random_matrix(n, 9)
    src = torch.from_numpy(np.ascontiguousarray(half.T)).cuda()
    fp64 = _values(gpu, half, n, 0)  # (also makes the workspace)
    d, e = src.clone(), torch.zeros(2 * n, dtype=torch.float64, device="cuda")
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        d.copy_(src)
        rc = gpu.zquatev_values_device(2 * n, d.data_ptr(), 2 * n, e.data_ptr(),
                                       torch.cuda.current_stream().cuda_stream)
    assert rc == 0, _lib.last_error()
    for _ in range(2):
        e.zero_()
        graph.replay()
        torch.cuda.synchronize()
        assert np.array_equal(e[:n].cpu().numpy(), fp64)
