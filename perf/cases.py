"""Performance cases of the quaternion eigensolver: what its users call, at the sizes they call it with.

Every case goes through a public entry point of the package (the C ABI's Python
mirrors, the torch operators, the batch plan, the request server). An
eigenvector of a Kramers pair is defined only up to a unit quaternion, so a pass
that returns eigenvectors ends with the phase convention that a program which
stores, compares or restarts from them applies: the first component of every
pair real and positive (`fix_phase`; for a real tridiagonal, the first
component's sign). The solvers work in place, so a pass begins by building the
input in the buffer that the solve overwrites.
"""
from __future__ import annotations

import math

import numpy as np
import torch

import zquatev_gb300.torch_ops  # noqa: F401  (registers torch.ops.zquatev_gb300)
from zquatev_gb300 import _lib, solver
from zquatev_gb300.serve import Server

C128, F64 = torch.complex128, torch.float64


def listed():
    return [
        # one small matrix on the GPU, as a model code solves per site or per atom: latency only
        {"name": "solve_tiny", "kind": "solve", "n": 23, "pad": 0},
        # a small molecule through the torch operator, odd quaternion order
        {"name": "torch_small", "kind": "torch", "n": 127},
        # the drop-in call on host arrays (pinned, padded leading dimension, odd order): a mid-size molecule
        {"name": "host_mid", "kind": "host", "n": 1023, "pad": 4},
        # the headline size: a large relativistic basis set, resident on the GPU
        {"name": "solve_large", "kind": "solve", "n": 4096, "pad": 0},
        # orbital energies only
        {"name": "values_mid", "kind": "values", "n": 750},
        # the plain FP64 path, selected by callers who want its residual
        {"name": "fp64_mid", "kind": "fp64", "n": 384},
        # symmetry blocks or k-points of several sizes solved every iteration: one plan, replayed
        {"name": "plan_mixed", "kind": "plan", "lo": 8, "hi": 256, "groups": 8, "per": 40, "sizes": 1},
        # many small blocks handed over in one call
        {"name": "batch_small", "kind": "batch", "n": 19, "count": 2000},
        # an SCF iteration with near-degenerate orbitals: solve, then the density with thermal occupations
        {"name": "scf_clustered", "kind": "scf", "n": 600},
        # the tridiagonal divide and conquer on its own
        {"name": "stedc_mid", "kind": "stedc", "n": 3000},
        # an FP64-accurate overlap product X^H Y of two tall blocks
        {"name": "zgemm_mid", "kind": "zgemm", "m": 1500, "n": 1100, "k": 3000, "opa": 2, "opb": 0},
        # a service's queue of host requests of all sizes
        {"name": "serve_mixed", "kind": "serve", "lo": 8, "hi": 512, "groups": 8, "per": 5, "sizes": 2},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["solve", "solve", "torch", "host", "values", "fp64", "plan", "batch", "scf", "stedc", "zgemm",
                       "serve"])
    if kind == "solve":
        return {"kind": kind, "n": _log(rng, 4, 4000), "pad": rng.choice([0, 0, 1, 6])}
    if kind == "torch":
        return {"kind": kind, "n": _log(rng, 16, 2000)}
    if kind == "host":
        return {"kind": kind, "n": _log(rng, 16, 2000), "pad": rng.choice([0, 0, 3, 8])}
    if kind == "values":
        return {"kind": kind, "n": _log(rng, 16, 1200)}
    if kind == "fp64":
        return {"kind": kind, "n": _log(rng, 32, 800)}
    if kind == "plan":
        return {"kind": kind, "lo": 8, "hi": _log(rng, 32, 256), "groups": rng.randint(3, 8), "per": rng.randint(5, 40),
                "sizes": rng.randrange(1000)}
    if kind == "batch":
        return {"kind": kind, "n": _log(rng, 3, 96), "count": _log(rng, 50, 3000)}
    if kind == "scf":
        return {"kind": kind, "n": _log(rng, 100, 1200)}
    if kind == "stedc":
        return {"kind": kind, "n": _log(rng, 40, 4000)}
    if kind == "zgemm":
        return {"kind": kind, "m": _log(rng, 100, 3000), "n": _log(rng, 100, 3000), "k": _log(rng, 100, 4000),
                "opa": rng.choice([0, 1, 2, 3]), "opb": rng.choice([0, 1, 2, 3])}
    return {"kind": "serve", "lo": 8, "hi": _log(rng, 64, 512), "groups": rng.randint(3, 8), "per": rng.randint(2, 5),
            "sizes": rng.randrange(1000)}


def group_orders(case):
    """Quaternion orders of a mixed batch: log-uniform, the largest one always there."""
    r = np.random.default_rng(case["sizes"])
    u = np.exp(r.uniform(math.log(case["lo"]), math.log(case["hi"]), case["groups"] - 1))
    return [case["hi"]] + [int(x) for x in np.floor(u)]


# ------------------------------------------------------------------ inputs
def _gen(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed))
    return g


def _randn(shape, g):
    return torch.randn(shape, dtype=C128, device="cuda", generator=g) * math.sqrt(2.0)


def blocks(n, g, count=1):
    """A (Hermitian) and B (antisymmetric), (count, n, n): Gaussian entries."""
    x, y = _randn((count, n, n), g), _randn((count, n, n), g)
    return (x + x.mH) / 2, (y - y.mT) / 2


def full(a, b):
    """The full matrix (A -B*; B A*)."""
    return torch.cat([torch.cat([a, -b.conj()], -1), torch.cat([b, a.conj()], -1)], -2)


def left_half(a, b, ld):
    """(count, n, ld): row j of a matrix holds column j of [A; B] (column-major storage), zeros below."""
    n = a.shape[-1]
    h = torch.zeros((a.shape[0], n, ld), dtype=C128, device="cuda")
    h[..., :n] = a.mT
    h[..., n:2 * n] = b.mT
    return h


def clustered_blocks(n, g):
    """H = Q diag(l) Q^H with 20% of the spectrum in clusters of 8, gaps 1e-6, the rest uniform in [-10, 10]."""
    ncl = int(0.2 * n) // 8
    free = torch.rand(n - 8 * ncl, dtype=F64, device="cuda", generator=g) * 20 - 10
    base = torch.rand(ncl, 1, dtype=F64, device="cuda", generator=g) * 20 - 10
    lam = torch.cat([free, (base + 1e-6 * torch.arange(8, dtype=F64, device="cuda")).reshape(-1)])
    a, b = blocks(n, g)
    k = 1j * full(a, b)[0] / math.sqrt(n)                    # anti-Hermitian with the quaternion structure
    one = torch.eye(2 * n, dtype=C128, device="cuda")
    q = torch.linalg.solve(one - k, one + k)                 # its Cayley transform: quaternion unitary
    h = (q * torch.cat([lam, lam])) @ q.mH
    a = (h[:n, :n] + h[n:, n:].conj()) / 2
    b = (h[n:, :n] - h[:n, n:].conj()) / 2
    return ((a + a.mH) / 2)[None], ((b - b.mT) / 2)[None]


def matrices(case, seed):
    """The (A, B) pairs that a case's matrices are made of, one pair of stacks per group of equal sizes."""
    g = _gen(seed)
    if case["kind"] in ("plan", "serve"):
        return [blocks(n, g, case["per"]) for n in group_orders(case)]
    if case["kind"] == "batch":
        return [blocks(case["n"], g, case["count"])]
    if case["kind"] == "scf":
        return [clustered_blocks(case["n"], g)]
    return [blocks(case["n"], g)]


def tridiagonal(n, g):
    """The tridiagonal that a Gaussian quaternion matrix of order n reduces to (independent normal and chi entries)."""
    d = torch.randn(n, dtype=F64, device="cuda", generator=g)
    dof = 4.0 * torch.arange(n - 1, 0, -1, dtype=F64, device="cuda")
    # a chi variate by the Wilson-Hilferty cube: chi2 ~ dof (1 - 2/(9 dof) + z sqrt(2/(9 dof)))^3
    z = torch.randn(n - 1, dtype=F64, device="cuda", generator=g)
    c = 2.0 / (9.0 * dof)
    return d, torch.sqrt((dof * (1 - c + z * torch.sqrt(c)) ** 3).abs() / 2)


def zgemm_operands(case, seed):
    g = _gen(seed)
    rows_a, cols_a = (case["m"], case["k"]) if case["opa"] in (0, 3) else (case["k"], case["m"])
    rows_b, cols_b = (case["k"], case["n"]) if case["opb"] in (0, 3) else (case["n"], case["k"])
    return _randn((cols_a, rows_a), g), _randn((cols_b, rows_b), g)   # column-major: one row per column


def _pinned(shape, dtype):
    return torch.empty(shape, dtype=dtype, pin_memory=True)


def prepare(case, seed):
    kind = case["kind"]
    s = {"kind": kind, "case": case}
    if kind == "stedc":
        n = case["n"]
        d, e = tridiagonal(n, _gen(seed))
        s.update(d=d, e=e, lam=torch.empty(n, dtype=F64, device="cuda"), z=torch.empty(n, n, dtype=F64, device="cuda"))
        return s
    if kind == "zgemm":
        a, b = zgemm_operands(case, seed)
        s.update(a=a, b=b, c=torch.empty(case["n"], case["m"], dtype=C128, device="cuda"))
        return s
    pairs = matrices(case, seed)
    if kind in ("torch", "values"):
        a, b = pairs[0]
        s["h"] = torch.cat([a[0], b[0]])
        return s
    if kind in ("plan", "batch"):
        shapes = [(a.shape[0], 2 * a.shape[-1]) for a, _ in pairs]
        n2s = np.repeat([n2 for _, n2 in shapes], [c for c, _ in shapes]).astype(np.int32)
        offs = np.concatenate([[0], np.cumsum(n2s.astype(np.int64) ** 2)])
        eoffs = np.concatenate([[0], np.cumsum(n2s.astype(np.int64))])
        d = torch.empty(int(offs[-1]), dtype=C128, device="cuda")
        eig = torch.zeros(int(eoffs[-1]), dtype=F64, device="cuda")
        s.update(d=d, eig=eig, views=[], halves=[left_half(a, b, 2 * a.shape[-1]) for a, b in pairs])
        i = 0
        for c, n2 in shapes:
            s["views"].append((d[int(offs[i]):int(offs[i + c])].view(c, n2, n2),
                               eig[int(eoffs[i]):int(eoffs[i + c])].view(c, n2)))
            i += c
        args = (n2s, n2s.copy(), offs[:-1].copy(), eoffs[:-1].copy())
        if kind == "plan":
            s["plan"] = solver.BatchPlan(*args)
        else:
            s["args"] = args
        return s
    if kind in ("host", "serve"):
        s.update(inputs=[], arrays=[], eigs=[])
        for a, b in pairs:
            c, n2 = a.shape[0], 2 * a.shape[-1]
            ld = n2 + case.get("pad", 0)
            half = _pinned((c, n2 // 2, ld), C128)
            half.copy_(left_half(a, b, ld))
            s["inputs"].append(half)
            s["arrays"].append(_pinned((c, n2, ld), C128).zero_())
            s["eigs"].append(_pinned((c, n2), F64).zero_())
        if kind == "serve":
            s["server"] = Server(hbm_budget_bytes=16 << 30)
        return s
    a, b = pairs[0]
    n = a.shape[-1]
    ld = 2 * n + case.get("pad", 0)
    s.update(half=left_half(a, b, ld)[0], d=torch.zeros(2 * n, ld, dtype=C128, device="cuda"),
             eig=torch.zeros(2 * n, dtype=F64, device="cuda"))
    if kind == "scf":
        s["p"] = torch.empty(2 * n, 2 * n, dtype=C128, device="cuda")
    return s


# -------------------------------------------------------------------- passes
def fix_phase(left, right, first_a, first_b):
    """Each column pair times the unit quaternion that makes its first component real and positive.

    first_a, first_b: rows 0 and n of the left columns, shaped to broadcast over them."""
    r = torch.rsqrt(first_a.abs().square() + first_b.abs().square())
    pa, pb = first_a.conj() * r, first_b * -r
    return (torch.addcmul(left * pa, right, pb), torch.addcmul(right * pa.conj(), left, -pb.conj()))


def fixed_columns(d, n2):
    """fix_phase for column-major storage: d (..., n2, ld), one row per column."""
    n = n2 // 2
    left, right = d[..., :n, :n2], d[..., n:, :n2]
    return fix_phase(left, right, left[..., :1], left[..., n:n + 1])


def occupations(eig):
    return torch.sigmoid(-eig / 0.5)


def run(s):
    kind = s["kind"]
    lib = _lib.load()
    stream = torch.cuda.current_stream().cuda_stream
    if kind == "solve":
        n2 = s["d"].shape[0]
        s["d"][: n2 // 2].copy_(s["half"])
        _lib.check(solver.zquatev_device(s["d"], s["eig"]), "zquatev_device")
        return (s["eig"][: n2 // 2], *fixed_columns(s["d"], n2))
    if kind == "fp64":
        n2 = s["d"].shape[0]
        s["d"][: n2 // 2].copy_(s["half"])
        _lib.check(lib.zquatev_fp64_device(n2, s["d"].data_ptr(), n2, s["eig"].data_ptr(), stream),
                   "zquatev_fp64_device")
        return (s["eig"][: n2 // 2], *fixed_columns(s["d"], n2))
    if kind == "torch":
        eig, v = torch.ops.zquatev_gb300.zquatev(s["h"])
        n = eig.numel()
        return (eig, *fix_phase(v[:, :n], v[:, n:], v[:1, :n], v[n:n + 1, :n]))
    if kind == "values":
        return torch.ops.zquatev_gb300.eigvalsh(s["h"])
    if kind in ("plan", "batch"):
        for half, (d, _) in zip(s["halves"], s["views"]):
            d[:, : d.shape[1] // 2].copy_(half)
        if kind == "plan":
            s["plan"].run(s["d"], s["eig"])
        else:
            n2s, ld2s, offs, eoffs = (x.ctypes.data for x in s["args"])
            _lib.check(lib.zquatev_batched_device(len(s["args"][0]), n2s, ld2s, offs, eoffs, s["d"].data_ptr(),
                                                  s["eig"].data_ptr(), stream), "zquatev_batched_device")
        return [(e[:, : e.shape[1] // 2], *fixed_columns(d, d.shape[1])) for d, e in s["views"]]
    if kind in ("host", "serve"):
        for half, d in zip(s["inputs"], s["arrays"]):
            d[:, : half.shape[1]].copy_(half)
        calls = [(d[i].numpy().T, e[i].numpy()) for d, e in zip(s["arrays"], s["eigs"]) for i in range(d.shape[0])]
        if kind == "host":
            for d, e in calls:
                _lib.check(solver.zquatev(d.shape[1], d, d.shape[0], e), "zquatev")
        else:
            ids = [s["server"].submit(d.shape[1], d, d.shape[0], e) for d, e in calls]
            for i in ids:
                _lib.check(s["server"].wait(i)[0], "request")
        # the eigenvectors go to the GPU, where the program that asked for them goes on
        return [(e[:, : e.shape[1] // 2], *fixed_columns(d.cuda(), d.shape[1]))
                for d, e in zip(s["arrays"], s["eigs"])]
    if kind == "scf":
        d, p, n2 = s["d"], s["p"], s["d"].shape[0]
        d[: n2 // 2].copy_(s["half"])
        _lib.check(solver.zquatev_device(d, s["eig"]), "zquatev_device")
        eig = s["eig"][: n2 // 2]
        w = d * occupations(torch.cat([eig, eig]))[:, None]
        _lib.check(lib.zq_zgemm_accurate(0, 2, n2, n2, n2, w.data_ptr(), n2, d.data_ptr(), n2, p.data_ptr(), n2,
                                         stream), "zq_zgemm_accurate")
        return eig, p
    if kind == "stedc":
        _lib.check(solver.stedc_device(s["d"], s["e"], s["lam"], s["z"]), "zq_stedc_device")
        return s["lam"], s["z"] * torch.sign(s["z"][:, :1])
    a, b, c, case = s["a"], s["b"], s["c"], s["case"]
    _lib.check(lib.zq_zgemm_accurate(case["opa"], case["opb"], case["m"], case["n"], case["k"], a.data_ptr(),
                                     a.shape[1], b.data_ptr(), b.shape[1], c.data_ptr(), case["m"], stream),
               "zq_zgemm_accurate")
    return c


# ------------------------------------------------------------ work and truth
def work(case):
    kind = case["kind"]
    if kind == "zgemm":
        m, n, k = case["m"], case["n"], case["k"]
        return {"bytes": 16.0 * (m * k + k * n + m * n), "flops": 8.0 * m * n * k}
    if kind == "stedc":
        n = case["n"]
        return {"bytes": 8.0 * (n * n + 3 * n), "flops": 4.0 / 3.0 * n ** 3}
    if kind in ("plan", "serve"):
        orders = group_orders(case) * case["per"]
    else:
        orders = [case["n"]] * case.get("count", 1)
    # reduction (64/3) n^3; the eigenvectors' way back through n quaternion reflectors 32 n^3
    vectors = kind != "values"
    nbytes = sum(32.0 * n * n + 8 * n + (64.0 * n * n if vectors else 0.0) for n in orders)
    flops = sum((64.0 / 3.0 + (32.0 if vectors else 0.0)) * n ** 3 for n in orders)
    if kind == "scf":
        n2 = 2 * case["n"]
        nbytes, flops = nbytes, flops + 8.0 * n2 ** 3 / 2
    return {"bytes": nbytes, "flops": flops}


def exact_pairs(a, b, columns_first):
    """Eigenvalues and phase-fixed eigenvectors of a stack of (A, B), by a dense Hermitian eigensolver."""
    n = a.shape[-1]
    w, v = torch.linalg.eigh(full(a, b))
    c = v[..., ::2]                                   # one vector of each Kramers pair; its partner is J c*
    partner = torch.cat([-c[..., n:, :].conj(), c[..., :n, :].conj()], -2)
    left, right = fix_phase(c, partner, c[..., :1, :], c[..., n:n + 1, :])
    if columns_first:
        left, right = left.mT.contiguous(), right.mT.contiguous()
    return (w[..., ::2] + w[..., 1::2]) / 2, left, right


def exact(case, seed):
    kind = case["kind"]
    if kind == "zgemm":
        a, b = zgemm_operands(case, seed)
        op = [lambda x: x.mT, lambda x: x, lambda x: x.conj(), lambda x: x.mH]    # of the column-major operand
        return (op[case["opa"]](a) @ op[case["opb"]](b)).mT.contiguous()
    if kind == "stedc":
        d, e = tridiagonal(case["n"], _gen(seed))
        w, v = torch.linalg.eigh(torch.diag(d) + torch.diag(e, 1) + torch.diag(e, -1))
        z = v.mT
        return w, z * torch.sign(z[:, :1])
    if case.get("n", 0) > 1500:
        return None
    pairs = matrices(case, seed)
    if kind == "values":
        w = torch.linalg.eigvalsh(full(*pairs[0])[0])
        return (w[::2] + w[1::2]) / 2
    if kind == "scf":
        w, v = torch.linalg.eigh(full(*pairs[0])[0])
        lam = (w[::2] + w[1::2]) / 2
        return lam, ((v * occupations(w)) @ v.mH).mT.contiguous()
    if kind == "torch":
        return tuple(x[0] for x in exact_pairs(*pairs[0], False))
    got = [exact_pairs(a, b, True) for a, b in pairs]
    if kind in ("solve", "fp64"):
        return tuple(x[0] for x in got[0])
    if kind == "host" or kind == "serve":
        return [(w.cpu(), left, right) for w, left, right in got]
    return got
