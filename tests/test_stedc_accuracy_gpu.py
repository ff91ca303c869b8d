"""The divide and conquer is as accurate as with FP64 merges, divisions and starting
values throughout: eigenvalues of a Toeplitz tridiagonal (known exactly; its halves are
equal, so that poles coincide), orthogonality of localised (Wilkinson) and of spread
eigenvectors. Orthogonality is formed exactly, from slices of 18 bits.

The bounds lie between what that algorithm gives and what an FP32 starting value in
small nodes, merges cut to 55 bits and products with reciprocals in zhat gave. Root mean
squares: of the eigenvalue errors over the norm 1.0e-16 to 1.2e-16 against 3.1e-16 to
3.3e-16 (their maxima are a few units of 1.1e-16 either way); of Z^T Z - I 1.7e-17
against 2.6e-17 (Wilkinson, n = 1200) and 7.2e-17 to 8.2e-17 against 7.9e-17 to 9.1e-17
(Gaussian)."""
import pytest

from zquatev_gb300 import _lib, solver

pytestmark = pytest.mark.gpu


def _solve(d, e):
    import torch

    n = d.numel()
    lam, z = torch.zeros_like(d), torch.zeros(n, n, dtype=d.dtype, device="cuda")
    assert solver.stedc_device(d, e, lam, z) == 0, _lib.last_error()
    return lam, z   # row j of z: eigenvector j


def _orthogonality(z):
    """Root mean square of Z Z^T - I: z cut into four slices of 18 bits, whose products are exact."""
    import torch

    n = z.shape[0]
    rest, cut = z.clone(), []
    for i in range(4):
        s = 2.0 ** (18 * (i + 1))
        cut.append(torch.trunc(rest * s))
        rest = rest - cut[-1] / s
    hi, lo = -torch.eye(n, dtype=z.dtype, device="cuda"), torch.zeros(n, n, dtype=z.dtype, device="cuda")
    for i in range(4):
        for j in range(min(4, 5 - i)):
            p = (cut[i] @ cut[j].T) * 2.0 ** (-18 * (i + j + 2))
            s = hi + p
            t = s - hi
            hi, lo = s, lo + ((hi - (s - t)) + (p - t))
    return (hi + lo).square().mean().sqrt().item()


@pytest.mark.parametrize("n", [40, 599, 600])
def test_eigenvalues_of_a_toeplitz_matrix(gpu, n):
    import numpy as np
    import torch

    lam, _ = _solve(torch.full((n,), 2.0, dtype=torch.float64, device="cuda"),
                    torch.ones(n - 1, dtype=torch.float64, device="cuda"))
    k = np.arange(1, n + 1)
    exact = 4 * np.sin(k * np.pi / (2 * (n + 1))) ** 2
    assert np.sqrt(np.mean((lam.cpu().numpy() - exact) ** 2)) <= 2.2e-16 * 4


def test_localised_eigenvectors(gpu):
    import torch

    n = 1200
    d = (torch.arange(n, dtype=torch.float64, device="cuda") - (n - 1) / 2).abs()
    _, z = _solve(d, torch.ones(n - 1, dtype=torch.float64, device="cuda"))
    assert _orthogonality(z) <= 2.1e-17


@pytest.mark.parametrize("n, bound", [(384, 8.6e-17), (599, 8.4e-17), (1200, 7.5e-17)])
def test_spread_eigenvectors(gpu, n, bound):
    import torch

    g = torch.Generator(device="cuda").manual_seed(1)
    d = torch.randn(n, dtype=torch.float64, device="cuda", generator=g)
    dof = 4.0 * torch.arange(n - 1, 0, -1, dtype=torch.float64, device="cuda")
    x = torch.randn(n - 1, dtype=torch.float64, device="cuda", generator=g)
    c = 2 / (9 * dof)
    _, z = _solve(d, torch.sqrt((dof * (1 - c + x * torch.sqrt(c)) ** 3).abs() / 2))
    assert _orthogonality(z) <= bound
