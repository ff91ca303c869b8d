"""The server's joint batches take their scratch from the device's stream-ordered pool,
like its other memory, and hold none of it once their requests have finished."""
import ctypes

import numpy as np
import pytest

from zquatev_gb300 import _lib, inputs
from zquatev_gb300.serve import Server

pytestmark = pytest.mark.gpu

RESERVED, USED = 5, 7   # cudaMemPoolAttrReservedMemCurrent, cudaMemPoolAttrUsedMemCurrent


def _pool(attr):
    """A figure of the device's default memory pool, from the runtime that the library loaded."""
    rt = ctypes.CDLL(_lib.LIB_PATH)
    pool, value = ctypes.c_void_p(), ctypes.c_uint64()
    assert rt.cudaDeviceGetDefaultMemPool(ctypes.byref(pool), 0) == 0
    assert rt.cudaMemPoolGetAttribute(pool, attr, ctypes.byref(value)) == 0
    return value.value


def _outside():
    """Device memory in use that is not the pool's."""
    import torch

    torch.cuda.synchronize()
    free, total = torch.cuda.mem_get_info()
    return total - free - _pool(RESERVED)


def _serve(srv, orders):
    ds = [np.array(inputs.random_matrix(n, i), order="F", copy=True) for i, n in enumerate(orders)]
    es = [np.zeros(n) for n in orders]
    ids = [srv.submit(2 * n, d, 2 * n, e) for n, d, e in zip(orders, ds, es)]
    assert [srv.wait(i)[0] for i in ids] == [0] * len(orders)


def test_scratch_comes_from_the_pool_and_goes_back(gpu):
    with Server(hbm_budget_bytes=4 << 30, batch_max_n2=512) as srv:
        _serve(srv, [20, 40, 9])        # modules, streams
        outside, used = _outside(), _pool(USED)
        _serve(srv, [200] * 20 + [64, 33] * 4)
        assert _outside() - outside <= 4 << 20
        assert _pool(USED) <= used
