"""A device-side wait of the FP64 path that runs out is reported: -104 from the
calls that wait for the GPU, eigenvalues that are not numbers from those that
do not; the context stays usable and the next call is correct.

The limit (300 cycles) is below one pass of the reduction's barrier through L2, at
an order whose group is not one cluster (a cluster's barrier has no limit)."""
import numpy as np
import pytest

from zquatev_gb300 import _lib, inputs
from zquatev_gb300.serve import Server

pytestmark = pytest.mark.gpu

N = 100
TIMEOUT = -104


@pytest.fixture
def short_wait(gpu):
    assert gpu.zq_set_pipeline_wait(300) == 0
    yield
    gpu.zq_set_pipeline_wait(0)


def _host(gpu, name, n):
    d = np.array(inputs.random_matrix(n, 7), order="F", copy=True)
    e = np.zeros(n)
    rc = getattr(gpu, name)(2 * n, d.ctypes.data, 2 * n, e.ctypes.data)
    return rc, e


def _reference(n):
    d = inputs.random_matrix(n, 7)
    return np.linalg.eigvalsh(inputs.full_from_blocks(d[:n, :n], d[n:, :n]))[::2]


@pytest.mark.parametrize("name, n", [("zquatev_c", N), ("zquatev_fp64_c", N), ("zquatev_values", N),
                                     ("zquatev_fp64_c", 1200)])
def test_host_calls_report_it(gpu, short_wait, name, n):
    rc, _ = _host(gpu, name, n)
    assert rc == TIMEOUT, rc
    assert "ran out of time" in _lib.last_error()
    gpu.zq_set_pipeline_wait(0)
    rc, e = _host(gpu, name, n)
    ref = _reference(n)
    assert rc == 0 and np.abs(e - ref).max() <= 1e-12 * np.abs(ref).max()


@pytest.mark.parametrize("name", ["zquatev_fp64_device", "zquatev_values_device"])
def test_asynchronous_calls_leave_no_numbers(gpu, short_wait, name):
    import torch

    h = torch.from_numpy(np.ascontiguousarray(inputs.random_matrix(N, 7).T)).cuda()
    st = torch.cuda.current_stream().cuda_stream
    for limit in (300, 0):
        gpu.zq_set_pipeline_wait(limit)
        d, e = h.clone(), torch.zeros(N, dtype=torch.float64, device="cuda")
        assert getattr(gpu, name)(2 * N, d.data_ptr(), 2 * N, e.data_ptr(), st) == 0
        e = e.cpu().numpy()
        if limit:
            assert np.isnan(e).all()
    ref = _reference(N)
    assert np.abs(e - ref).max() <= 1e-12 * np.abs(ref).max()


def test_large_matrices_of_a_batch(gpu, short_wait):
    import torch

    orders = [300, 5, 270]
    n2 = np.array([2 * n for n in orders], np.int32)
    offs = np.concatenate([[0], np.cumsum(n2.astype(np.int64) ** 2)])
    eoffs = np.concatenate([[0], np.cumsum(n2.astype(np.int64))])
    host = np.concatenate([inputs.random_matrix(n, 7).ravel(order="F") for n in orders])
    for limit, want in ((300, TIMEOUT), (0, 0)):
        gpu.zq_set_pipeline_wait(limit)
        d = torch.from_numpy(host).cuda()
        e = torch.zeros(int(eoffs[-1]), dtype=torch.float64, device="cuda")
        rc = gpu.zquatev_batched_device(3, n2.ctypes.data, n2.ctypes.data, offs.ctypes.data, eoffs.ctypes.data,
                                        d.data_ptr(), e.data_ptr(), torch.cuda.current_stream().cuda_stream)
        assert rc == want


def test_server_lane(gpu, short_wait):
    assert gpu.zq_set_path(0) == 0
    try:
        with Server(lanes=1, batch_max_n2=0) as srv:
            for limit, want in ((300, TIMEOUT), (0, 0)):
                gpu.zq_set_pipeline_wait(limit)
                d = np.array(inputs.random_matrix(N, 7), order="F", copy=True)
                assert srv.wait(srv.submit(2 * N, d, 2 * N, np.zeros(N)))[0] == want
    finally:
        gpu.zq_set_path(2)
