"""GPU tests of the batched Q formation (zq_backtransform.cu) through the refined path:
orders at the edges of its blocks of 64 reflectors, with even and odd numbers of rows,
of one chunk of Gram sums and of the scratch it needs (below order ~35 the general
formation runs).

Tolerance: the parity suite's 1e-12 on the result; and the FP32 start must be good
enough for the refinement to converge by itself (no FP64 fallback).
"""
import numpy as np
import pytest

from zquatev_gb300 import inputs, metrics, solver

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [3, 20, 34, 40, 65, 66, 67, 68, 129, 130, 131, 194, 255, 256, 257, 322, 515])
def test_refined_from_its_q(gpu, n):
    d = inputs.random_matrix(n, 60 + n)
    out = np.array(d, order="F", copy=True)
    eig = np.zeros(2 * n)
    assert solver.zquatev_refined(2 * n, out, 2 * n, eig) == 0
    assert not solver.refine_stats()[2]
    h = inputs.full_from_blocks(d[:n, :n], d[n:, :n])
    ref = np.linalg.eigvalsh(h)[::2]
    assert metrics.eig_error(eig[:n], ref, metrics.h_norm2(ref)) <= 1e-12
    assert metrics.residual(h, out, eig[:n]) <= 1e-12
    assert metrics.orthonormality(out) <= 1e-12


@pytest.mark.parametrize("path", ["refined", "auto"])
def test_uncoupled_equal_eigenvalues(gpu, path):
    """Equal Rayleigh quotients whose coupling is exactly zero: no correction, no reciprocal of the zero gap."""
    n = 300
    lam = np.repeat(np.arange(30.0), 10) - 3.0
    d = np.zeros((2 * n, 2 * n), np.complex128, order="F")
    d[:n, :n] = np.diag(np.random.default_rng(2).permutation(lam))
    h = inputs.full_from_blocks(d[:n, :n], d[n:, :n])
    eig = np.zeros(2 * n)
    fn = solver.zquatev_refined if path == "refined" else solver.zquatev
    assert fn(2 * n, d, 2 * n, eig) == 0
    assert np.abs(eig[:n] - np.sort(lam)).max() <= 1e-12 * 30
    assert metrics.residual(h, d, eig[:n]) <= 1e-12
    assert metrics.orthonormality(d) <= 1e-12
