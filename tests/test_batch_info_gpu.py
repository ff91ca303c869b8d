"""A matrix whose tridiagonal solve does not come to an end (it holds a value that is
not a number) is counted in the batch's info, whichever way its order is solved, and
leaves the others alone."""
import numpy as np
import pytest

from zquatev_gb300 import _lib, inputs, solver
from zquatev_gb300.serve import Server

pytestmark = pytest.mark.gpu


def _batch(orders, bad):
    import torch

    n2 = np.array([2 * n for n in orders], np.int32)
    offs = np.concatenate([[0], np.cumsum(n2.astype(np.int64) ** 2)[:-1]])
    eoffs = np.concatenate([[0], np.cumsum(np.array(orders, np.int64))[:-1]])
    mats = [inputs.random_matrix(n, 20 + i) for i, n in enumerate(orders)]
    for i, v in bad.items():
        mats[i][orders[i] // 2, orders[i] // 2] = v
    return mats, torch.from_numpy(np.concatenate([m.ravel(order="F") for m in mats])).cuda(), \
        torch.zeros(sum(orders), dtype=torch.float64, device="cuda"), (n2, n2.copy(), offs, eoffs)


def _good(orders, mats, eig, bad):
    at = 0
    for i, (n, m) in enumerate(zip(orders, mats)):
        w = eig[at:at + n]
        at += n
        if i in bad:
            assert not np.isfinite(w).all()
            continue
        ref = np.linalg.eigvalsh(inputs.full_from_blocks(m[:n, :n], m[n:, :n]))[::2]
        assert np.abs(w - ref).max() <= 1e-12 * np.abs(ref).max()


ORDERS = [200, 90, 40, 20, 9]


@pytest.mark.parametrize("which", range(len(ORDERS)))
@pytest.mark.parametrize("value", [float("nan"), float("inf")])
@pytest.mark.parametrize("entry", ["batch", "plan", "server"])
def test_counted(gpu, entry, which, value):
    import torch

    bad = {which: value}
    mats, d, e, args = _batch(ORDERS, bad)
    if entry == "batch":
        info = gpu.zquatev_batched_device(len(ORDERS), *(a.ctypes.data for a in args), d.data_ptr(), e.data_ptr(), 0)
        assert info > 0, (info, _lib.last_error())
    elif entry == "plan":
        plan = solver.BatchPlan(*args, ctas_per_sm=1)
        plan.run(d, e)
        assert plan.info() > 0
        plan.close()
    else:
        with Server(hbm_budget_bytes=1 << 30, batch_max_n2=512) as srv:
            work, eigs = [np.array(m, order="F", copy=True) for m in mats], [np.zeros(n) for n in ORDERS]
            ids = [srv.submit(2 * n, w, 2 * n, x) for n, w, x in zip(ORDERS, work, eigs)]
            infos = [srv.wait(i)[0] for i in ids]
        assert infos[which] > 0 and not any(infos[:which] + infos[which + 1:]), infos
        _good(ORDERS, mats, np.concatenate(eigs), bad)
        return
    torch.cuda.synchronize()
    _good(ORDERS, mats, e.cpu().numpy(), bad)
