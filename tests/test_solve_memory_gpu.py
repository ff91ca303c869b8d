"""Solves whose best workspace (with the residues of the products and of the merges)
does not fit run in the least one; the server admits a request by it where the best
exceeds its whole budget."""
import contextlib
import gc

import numpy as np
import pytest

from zquatev_gb300 import _lib, inputs
from zquatev_gb300.serve import Server

pytestmark = pytest.mark.gpu

MB = 1 << 20


def _free():
    import torch

    gc.collect()
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    return torch.cuda.mem_get_info()[0]


@contextlib.contextmanager
def _crowded(leave):
    import torch

    ballast = torch.empty(_free() - leave, dtype=torch.uint8, device="cuda")
    try:
        yield
    finally:
        del ballast
        _free()


def _matrix_bytes(n):
    return 64 * n * n + 8 * (n + 32)


def _check(h, d, e, n):
    import torch

    v, w = d.T, e[:n]
    norm = w.abs().max()
    hv = h @ v
    assert ((hv - v * torch.cat([w, w])).abs().max() / norm).item() <= 1e-12
    assert (v.mH @ v - torch.eye(2 * n, dtype=v.dtype, device="cuda")).abs().max().item() <= 1e-12


@pytest.mark.parametrize("entry, short", [("fp64", 60 * MB), ("refined", 800 * MB)])
def test_solve_in_the_least_workspace(gpu, entry, short):
    """n = 2000: the merges' residues take 130 MB, the products' 1.7 GB (digits 0.5 GB)."""
    import torch

    n = 2000
    st = torch.cuda.current_stream().cuda_stream

    def solve(d, e):
        if entry == "fp64":
            return gpu.zquatev_fp64_device(2 * n, d.data_ptr(), 2 * n, e.data_ptr(), st)
        return gpu.zquatev_refined_device(2 * n, d.data_ptr(), 2 * n, e.data_ptr(), st, 1)

    gpu.zq_release_workspace()
    m = inputs.random_matrix(n, 17)
    h = torch.from_numpy(inputs.full_from_blocks(m[:n, :n], m[n:, :n])).cuda()
    d0 = torch.from_numpy(np.ascontiguousarray(m.T)).cuda()
    small, es = torch.zeros(40, 40, dtype=torch.complex128, device="cuda"), torch.zeros(20, dtype=torch.float64, device="cuda")
    assert gpu.zquatev_fp64_device(40, small.data_ptr(), 40, es.data_ptr(), st) == 0      # modules and streams
    d, e = d0.clone(), torch.zeros(n, dtype=torch.float64, device="cuda")
    need = gpu.zq_solve_footprint(2 * n, 1 if entry == "refined" else 0) - _matrix_bytes(n)
    with _crowded(need - short):
        rcs = [solve(d, e)]
        d.copy_(d0)
        rcs.append(solve(d, e))           # and again in what the first call left
        torch.cuda.synchronize()
        gpu.zq_release_workspace()
    assert rcs == [0, 0], (rcs, _lib.last_error())
    _check(h, d, e, n)


def test_server_admits_by_the_least(gpu):
    n = 600
    budget = gpu.zq_solve_footprint(2 * n, 1) - 60 * MB
    m = inputs.random_matrix(n, 3)
    d, e = np.array(m, order="F", copy=True), np.zeros(n)
    with Server(hbm_budget_bytes=budget, lanes=1) as srv:
        info, t = srv.wait(srv.submit(2 * n, d, 2 * n, e))
        assert info == 0 and t["path"] == "refined"
        assert srv.stats()["peak_reserved_bytes"] <= budget
    h = inputs.full_from_blocks(m[:n, :n], m[n:, :n])
    norm = np.abs(e).max()
    assert np.abs(h @ d - d * np.concatenate([e, e])).max() <= 1e-12 * norm
    assert np.abs(d.conj().T @ d - np.eye(2 * n)).max() <= 1e-12
