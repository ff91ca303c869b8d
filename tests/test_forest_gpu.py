"""GPU tests of the mid-size batch path (zq_forest.cu): orders at the edges of
its range, of the reduction's classes and of the back-transform's row classes,
with padded leading dimensions, in batches with few and with many columns (a CTA
or a warp per column) and mixed with matrices of the other paths; replays of a
plan; a second layout through the same workspace.

Tolerance: the bars of the parity suite (1e-12 relative to ||H||_2).
"""
import numpy as np
import pytest

from zquatev_gb300 import _lib, inputs, solver

pytestmark = pytest.mark.gpu

TOL = 1e-12
ORDERS = [256, 255, 225, 224, 193, 192, 161, 160, 129, 128, 97, 96, 65, 64, 63, 34, 33, 32, 31, 1, 0]


def _batch(orders, seed):
    import torch

    lds = [2 * n + (i % 3) for i, n in enumerate(orders)]
    offs, at = [], 5
    for n, ld in zip(orders, lds):
        offs.append(at)
        at += 2 * n * ld + 3
    host = np.full(at, np.nan + 0j)
    for i, (n, ld, o) in enumerate(zip(orders, lds, offs)):
        host[o:o + 2 * n * ld] = inputs.random_matrix(n, seed + i, ld2=ld).ravel(order="F") if n else 0
    eoffs = np.concatenate([[0], np.cumsum([n + 1 for n in orders])[:-1]]).astype(np.int64)
    args = (np.array([2 * n for n in orders], np.int32), np.array(lds, np.int32), np.array(offs, np.int64), eoffs)
    return torch.from_numpy(host).cuda(), int(sum(n + 1 for n in orders)), args


def _check(orders, args, before, after, eig):
    import torch

    for n, ld, o, eo in zip(orders, *(a.tolist() for a in args[1:])):
        if n == 0:
            continue
        h0 = before[o:o + 2 * n * ld].view(2 * n, ld)[:, : 2 * n].T
        v = after[o:o + 2 * n * ld].view(2 * n, ld)[:, : 2 * n].T
        a, b = h0[:n, :n], h0[n:, :n]
        h = torch.cat([torch.cat([a, -b.conj()], 1), torch.cat([b, a.conj()], 1)])
        w = eig[eo:eo + n]
        norm = w.abs().max()
        assert (w.diff() >= 0).all()
        assert ((h @ v - v * torch.cat([w, w])).abs().max() / norm).item() <= TOL
        assert (v.mH @ v - torch.eye(2 * n, dtype=v.dtype, device=v.device)).abs().max().item() <= TOL
        assert torch.equal(v[:n, n:], -v[n:, :n].conj()) and torch.equal(v[n:, n:], v[:n, :n].conj())
        assert (eig[eo + n] == -3.0).item()
    ends = [o + 2 * n * ld for n, ld, o in zip(orders, args[1].tolist(), args[2].tolist())]
    for e in ends:  # the gaps between the matrices are untouched
        assert torch.isnan(after[e:e + 3].real).all()


@pytest.mark.parametrize("copies", [1, 6])
def test_batched_orders(gpu, copies):
    import torch

    orders = ORDERS * copies
    d0, ne, args = _batch(orders, 40)
    d, e = d0.clone(), torch.full((ne,), -3.0, dtype=torch.float64, device="cuda")
    rc = gpu.zquatev_batched_device(len(orders), *(a.ctypes.data for a in args), d.data_ptr(), e.data_ptr(),
                                    torch.cuda.current_stream().cuda_stream)
    assert rc == 0, _lib.last_error()
    _check(orders, args, d0, d, e)


def test_plan_of_mid_sizes_only(gpu):
    import torch

    orders = [40, 200, 100]
    d0, ne, args = _batch(orders, 90)
    plan = solver.BatchPlan(*args)
    for _ in range(3):
        d, e = d0.clone(), torch.full((ne,), -3.0, dtype=torch.float64, device="cuda")
        plan.run(d, e)
        assert plan.info() == 0
        _check(orders, args, d0, d, e)
    plan.close()


def test_layouts_share_the_workspace(gpu):
    import torch

    for orders in ([250, 60, 33], [90] * 20, [250, 60, 33]):
        d0, ne, args = _batch(orders, len(orders))
        d, e = d0.clone(), torch.full((ne,), -3.0, dtype=torch.float64, device="cuda")
        rc = gpu.zquatev_batched_device(len(orders), *(a.ctypes.data for a in args), d.data_ptr(), e.data_ptr(), 0)
        assert rc == 0, _lib.last_error()
        _check(orders, args, d0, d, e)


@pytest.mark.parametrize("orders", [[48], [64, 33, 32, 20, 16, 15, 3], [256, 130, 40] + [9] * 130])
def test_server_batches(gpu, orders):
    """Requests in allocations of their own, alone, with few and with many small ones beside them."""
    import torch

    from zquatev_gb300.serve import Server

    with Server(hbm_budget_bytes=4 << 30, batch_max_n2=512) as srv:
        for _ in range(2):
            before = [inputs.random_matrix(n, 700 + i) for i, n in enumerate(orders)]
            work = [np.array(d, order="F", copy=True) for d in before]
            eigs = [np.zeros(n) for n in orders]
            ids = [srv.submit(2 * n, d, 2 * n, e) for n, d, e in zip(orders, work, eigs)]
            for i in ids:
                info, t = srv.wait(i)
                assert info == 0 and t["path"] == "batched"
            for n, d0, d, w in zip(orders, before, work, eigs):
                h = inputs.full_from_blocks(d0[:n, :n], d0[n:, :n])
                lam = np.concatenate([w, w])
                assert (np.diff(w) >= 0).all()
                assert np.abs(h @ d - d * lam).max() <= TOL * np.abs(w).max()
                assert np.abs(d.conj().T @ d - np.eye(2 * n)).max() <= TOL
        assert srv.stats()["peak_reserved_bytes"] <= 4 << 30
