"""The joint solve's scratch: bounded by its largest part, and done without where
the device has no room for it."""
import contextlib
import gc

import numpy as np
import pytest

from zquatev_gb300 import _lib, inputs, solver

pytestmark = pytest.mark.gpu

MB = 1 << 20


def _copies(n, count, seed=3):
    import torch

    n2 = np.full(count, 2 * n, np.int32)
    offs = np.arange(count, dtype=np.int64) * (4 * n * n)
    eoffs = np.arange(count, dtype=np.int64) * n
    one = torch.from_numpy(np.ascontiguousarray(inputs.random_matrix(n, seed).T)).cuda()
    return one[None].repeat(count, 1, 1), torch.zeros(count, n, dtype=torch.float64, device="cuda"), (n2, n2.copy(), offs, eoffs)


def _run(gpu, d, e, args):
    import torch

    return gpu.zquatev_batched_device(len(args[0]), *(a.ctypes.data for a in args), d.data_ptr(), e.data_ptr(),
                                      torch.cuda.current_stream().cuda_stream)


def _check(n, d, e, seed=3):
    import torch

    m = inputs.random_matrix(n, seed)
    h = torch.from_numpy(inputs.full_from_blocks(m[:n, :n], m[n:, :n])).cuda()
    v, w = d[0].T, e[0]
    norm = w.abs().max()
    assert ((h @ v - v * torch.cat([w, w])).abs().max() / norm).item() <= 1e-12
    assert (v.mH @ v - torch.eye(2 * n, dtype=v.dtype, device="cuda")).abs().max().item() <= 1e-12
    assert (e == e[0]).all() and (d == d[0]).all()


def _free():
    import torch

    gc.collect()
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    return torch.cuda.mem_get_info()[0]


def test_parts_share_the_scratch(gpu, monkeypatch):
    """256 matrices of order 256 in eight parts: 3 x 16 MB of eigenvectors a part."""
    d, e, args = _copies(256, 256)
    assert _run(gpu, d[:1], e[:1], tuple(a[:1] for a in args)) == 0   # modules, streams
    gpu.zq_release_workspace()
    monkeypatch.setenv("ZQ_FOREST_CHUNK", str(1 << 21))
    d, e, args = _copies(256, 256)
    before = _free()
    assert _run(gpu, d, e, args) == 0, _lib.last_error()
    held = before - _free()
    _check(256, d, e)
    gpu.zq_release_workspace()
    assert held <= 150 * MB, held / MB


@pytest.mark.parametrize("entry", ["batch", "plan"])
def test_parts_of_mixed_orders(gpu, monkeypatch, entry):
    """Five orders in many parts, each part with tables of its own (the second pass reuses them)."""
    import torch

    monkeypatch.setenv("ZQ_FOREST_CHUNK", "40000")
    orders = sorted([200, 130, 64, 33, 97] * 7, reverse=True)
    n2 = np.array([2 * n for n in orders], np.int32)
    offs = np.concatenate([[0], np.cumsum(n2.astype(np.int64) ** 2)[:-1]])
    eoffs = np.concatenate([[0], np.cumsum(np.array(orders, np.int64))[:-1]])
    mats = [inputs.random_matrix(n, 40 + i) for i, n in enumerate(orders)]
    d0 = torch.from_numpy(np.concatenate([m.ravel(order="F") for m in mats])).cuda()
    args = (n2, n2.copy(), offs, eoffs)
    plan = solver.BatchPlan(*args) if entry == "plan" else None
    for _ in range(2):
        d, e = d0.clone(), torch.zeros(sum(orders), dtype=torch.float64, device="cuda")
        if plan:
            plan.run(d, e)
            assert plan.info() == 0
        else:
            assert _run(gpu, d, e, args) == 0, _lib.last_error()
        out, w = d.cpu().numpy(), e.cpu().numpy()
        for n, m, o, eo in zip(orders, mats, offs, eoffs):
            h = inputs.full_from_blocks(m[:n, :n], m[n:, :n])
            v = out[o:o + 4 * n * n].reshape(2 * n, 2 * n).T
            lam = w[eo:eo + n]
            norm = np.abs(lam).max()
            assert np.abs(h @ v - v * np.concatenate([lam, lam])).max() <= 1e-12 * norm
            assert np.abs(v.conj().T @ v - np.eye(2 * n)).max() <= 1e-12
    if plan:
        plan.close()
    gpu.zq_release_workspace()


@contextlib.contextmanager
def _crowded(leave):
    """The device's memory taken but for `leave` bytes."""
    import torch

    ballast = torch.empty(_free() - leave, dtype=torch.uint8, device="cuda")
    try:
        yield
    finally:
        del ballast
        _free()


def test_batch_without_room(gpu):
    """Three eigenvector buffers (400 MB) do not fit; the CTA kernel's 140 MB do."""
    d, e, args = _copies(256, 256)
    assert _run(gpu, d[:1].clone(), e[:1].clone(), tuple(a[:1] for a in args)) == 0
    gpu.zq_release_workspace()
    with _crowded(300 * MB):
        rc = _run(gpu, d, e, args)
    assert rc == 0, _lib.last_error()
    _check(256, d, e)


def test_plan_without_room(gpu):
    d, e, args = _copies(256, 256)
    gpu.zq_release_workspace()
    with _crowded(300 * MB):
        plan = solver.BatchPlan(*args, ctas_per_sm=1)
        plan.run(d, e)
        assert plan.info() == 0
        plan.close()
    _check(256, d, e)
