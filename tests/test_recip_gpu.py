"""The reciprocal and reciprocal square root of zq_recip.cuh over their stated ranges,
against their stated error bounds and against division and rsqrt.

Bounds: the functional iteration leaves out terms below 2^-60 (2^-58) and rounds once,
2^-53 relative (the square root's residual rounds q y too, another 2^-54); the bounds
allow 2^-6 of that for what is left out. A residual itself is off by less than 2^-100."""
import ctypes
import os
import subprocess

import pytest

from zquatev_gb300 import build

pytestmark = pytest.mark.gpu

HERE = os.path.dirname(os.path.abspath(__file__))
N = 1 << 22
EPS = 2.0 ** -53


@pytest.fixture(scope="module")
def math(gpu, tmp_path_factory):
    out = tmp_path_factory.mktemp("device_math") / "recip.so"
    cmd = [build._nvcc(), *build.ARCH, "-O3", "-std=c++17", "-Xcompiler", "-fPIC", "-shared", "-cudart", "shared",
           "-I" + build.CSRC, os.path.join(HERE, "device_math", "recip.cu"), "-o", str(out)]
    r = subprocess.run(cmd, capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    return ctypes.CDLL(str(out))


def _run(math, which, x):
    import torch

    y, err = torch.empty_like(x), torch.empty_like(x)
    torch.cuda.synchronize()
    rc = math.test_recip(which, *(ctypes.c_void_p(t.data_ptr()) for t in (x, y, err)), ctypes.c_longlong(x.numel()))
    assert rc == 0
    return y, err


def _inputs(lo, hi, seed):
    """Magnitudes spread over the exponents lo..hi, mantissas random and next to powers of two."""
    import torch

    g = torch.Generator(device="cuda").manual_seed(seed)
    m = 1 + torch.rand(N, dtype=torch.float64, device="cuda", generator=g)
    k = torch.arange(1, 5, dtype=torch.float64, device="cuda") * 2 ** -52
    m[:4], m[4:8], m[8] = 1 + k, 2 - 2 * k, 1.0
    e = torch.randint(lo, hi, (N,), device="cuda", generator=g)
    return torch.ldexp(m, e)


def test_recip(math):
    import torch

    x = _inputs(-1021, 1020, 1)
    x = torch.where(torch.arange(N, device="cuda") % 2 == 0, x, -x)
    y, err = _run(math, 0, x)
    assert err.abs().max().item() <= EPS * (1 + 2 ** -6)
    ulps = (y.view(torch.int64) - (1.0 / x).view(torch.int64)).abs()
    assert ulps.max().item() <= 1


def test_recip_sqrt(math):
    import torch

    x = _inputs(-900, 900, 2)
    y, err = _run(math, 1, x)
    assert err.abs().max().item() <= 1.5 * EPS * (1 + 2 ** -6)
    ulps = (y.view(torch.int64) - torch.rsqrt(x).view(torch.int64)).abs()
    assert ulps.max().item() <= 2   # each within one of the exact value


def test_recip_of_what_is_not_a_number(math):
    import torch

    x = torch.tensor([0.0, -0.0, float("inf"), float("-inf"), float("nan")], dtype=torch.float64, device="cuda")
    y, _ = _run(math, 0, x)
    assert torch.isnan(y).all()
