"""Performance cases of the batched complex eigensolver.

Each case is one pass of work that users have this library do, through the
entry points of the `ves` module, from the inputs to eigenpairs that can be
used.  `listed()` gives the fixed cases, `draw(rng)` more of the same ranges,
`prepare` what a program has in hand before the call, `run` one pass, `work`
the arithmetic and bytes the pass cannot do without, and `exact` the same
outputs from numpy in 64 bits.

Output convention.  A Schur form leaves the eigenvalues in the order in which
they deflated and the eigenvectors with arbitrary unit phases, so a program
that uses the eigenpairs brings them into a convention of its own.  Here: unit
2-norm (the library's own option), eigenvalues ascending by real part, and the
first component of every eigenvector real and positive.  It is part of `run`
(torch operations on the device), so that its outputs have a definite value.
"""
import math
import os
import sys

import numpy as np
import torch

_ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
_PKG = os.path.join(_ROOT, "vectorized-eigensolver_gb300")
if _PKG not in sys.path:
    sys.path.insert(0, _PKG)

import learned_shift  # noqa: E402
import ves  # noqa: E402

DEV = "cuda"


def listed():
    return [
        # one problem's worth of small matrices, as in the Python interface's
        # own examples (2 blocks of 4): the latency of a call
        {"name": "small-8", "kind": "solve", "n": 8, "bc": 2, "tc": 4, "prec": 0},
        # a call from a host program in NumPy arrays, at the reference's CPU size
        {"name": "host-8", "kind": "host", "n": 8, "bc": 2500, "tc": 4},
        # an odd order and an odd interleave, some tens of thousands of matrices
        {"name": "solve-13", "kind": "solve", "n": 13, "bc": 9, "tc": 1999, "prec": 0},
        # the main workload: a million 16x16 matrices in FP64
        {"name": "solve-16", "kind": "solve", "n": 16, "bc": 2048, "tc": 512, "prec": 0},
        # 32x32 in FP64
        {"name": "solve-32", "kind": "solve", "n": 32, "bc": 128, "tc": 512, "prec": 0},
        # a few hundred large matrices: fewer than the GPU has lanes
        {"name": "solve-57", "kind": "solve", "n": 57, "bc": 3, "tc": 100, "prec": 0},
        # eigenvalues without vectors (stability and spectrum scans)
        {"name": "values-24", "kind": "values", "n": 24, "bc": 60, "tc": 512},
        # the mixed-precision form at its two benchmark orders and an odd one
        {"name": "refine-9", "kind": "solve", "n": 9, "bc": 30, "tc": 1001, "prec": 1},
        {"name": "refine-16", "kind": "solve", "n": 16, "bc": 1024, "tc": 512, "prec": 1},
        {"name": "refine-32", "kind": "solve", "n": 32, "bc": 128, "tc": 512, "prec": 1},
        # one call over matrices of every order from 4 to 64
        {"name": "varsize", "kind": "varsize", "count": 20000, "nmin": 4, "nmax": 64},
        # a parametric family with a trained shift network: inference, polish,
        # shift-seeded FP64 solve
        {"name": "learned-24", "kind": "learned", "n": 24, "bc": 64, "tc": 512},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["solve", "solve", "refine", "refine", "values", "varsize", "host", "learned"])
    if kind == "varsize":
        nmin = rng.randint(2, 24)
        return {"kind": kind, "count": _log_int(rng, 50, 20000), "nmin": nmin, "nmax": rng.randint(nmin, 64)}
    n = rng.randint(8, 40) if kind == "learned" else _log_int(rng, 2, 64)
    # flops up to a quarter of the largest listed case's (for host buffers less)
    most = max(8, int(1_048_576 * 16 ** 3 / 4 / n ** 3))
    most = min(most, {"host": 60_000, "learned": 60_000}.get(kind, 400_000))
    N = _log_int(rng, 4096 if kind == "learned" else 1, max(most, 4096))
    tc = min(N, rng.choice([1, 4, 32, 37, 100, 512, N]))
    c = {"kind": "solve" if kind == "refine" else kind, "n": n, "bc": max(1, N // tc), "tc": tc}
    if kind in ("solve", "refine"):
        c["prec"] = int(kind == "refine")
    return c


def _gauss(g, *shape):
    return torch.complex(torch.randn(*shape, generator=g, dtype=torch.float64, device=DEV),
                         torch.randn(*shape, generator=g, dtype=torch.float64, device=DEV))


def _planes(count, k):
    return [torch.empty(count, dtype=torch.float64, device=DEV) for _ in range(k)]


def _varsize_inputs(case, seed):
    """Matrices of every order in [nmin, nmax] equally often, shuffled, every other
    one of an order Hermitian, packed one after another (column-major): dims,
    planes, and per order its matrices."""
    g = torch.Generator(device=DEV).manual_seed(seed)
    dims = case["nmin"] + torch.arange(case["count"], device=DEV) % (case["nmax"] - case["nmin"] + 1)
    dims = dims[torch.randperm(case["count"], generator=g, device=DEV)]
    aoff = torch.cumsum(dims * dims, 0) - dims * dims
    re, im = _planes(int((dims * dims).sum()), 2)
    groups = []
    for n in range(case["nmin"], case["nmax"] + 1):
        idx = torch.nonzero(dims == n)[:, 0]
        if not len(idx):
            continue
        A = _gauss(g, len(idx), n, n)
        A[::2] = (A[::2] + A[::2].mH) / 2
        pos = (aoff[idx][:, None] + torch.arange(n * n, device=DEV)).reshape(-1)
        cols = A.transpose(1, 2).reshape(-1)
        re[pos], im[pos] = cols.real, cols.imag
        groups.append((idx, A))
    return dims, re, im, groups


_nets = {}  # order -> the trained network that a program loads once


def prepare(case, seed):
    kind = case["kind"]
    s = dict(case)
    if kind == "varsize":
        dims, re, im, _ = _varsize_inputs(case, seed)
        ne, nm = int(dims.sum()), len(re)
        s["opt"] = ves.default_options(vnorm=ves.VNORM_TWO)
        s["dims"], s["A"] = dims.to(torch.int32), (re, im)
        s["E"], s["V"] = _planes(ne, 2), _planes(nm, 2)
        s["ws"] = ves.varsize_workspace(case["count"], case["nmax"], s["opt"])
        # where each eigenvalue's matrix and each vector component's column are
        s["mat"] = torch.repeat_interleave(torch.arange(len(dims), device=DEV), dims)
        n_of = torch.repeat_interleave(dims, dims)
        s["start"] = torch.cumsum(n_of, 0) - n_of
        s["col"] = torch.repeat_interleave(torch.arange(ne, device=DEV), n_of)
        s["row"] = torch.arange(nm, device=DEV) - s["start"][s["col"]]
        return s
    n, tc, N = case["n"], case["tc"], case["bc"] * case["tc"]
    if kind == "learned":
        if n not in _nets:
            _nets[n], _ = learned_shift.train(n, count=20_480, epochs=30, layers=3, loss=1, delta=0.01)
        s["net"] = _nets[n]
        s["p"], *s["A"] = learned_shift.family(N, n, param_seed=seed, thread_cnt=tc, device=DEV)
        s["opt"] = ves.default_options(vnorm=ves.VNORM_TWO, shift_sweeps=1, shift_polish=16, shift_gate=0.0)
        s["E"], s["V"], s["S"] = _planes(N * n, 2), _planes(N * n * n, 2), _planes(N * n, 2)
        s["ws"] = ves.shifts_workspace(n, case["bc"], tc, s["opt"])
        s["pws"] = s["net"].predict_workspace(N)
        s["Zv"], s["Ze"] = _complex_buffers(N, n)
        return s
    z = _gauss(torch.Generator(device=DEV).manual_seed(seed), N, n, n)
    if kind == "host":
        s["A"] = ves.soa_from_complex(z.cpu().numpy(), tc)
        s["T"] = [np.empty_like(a) for a in s["A"]]
        s["E"] = [np.empty(N * n) for _ in range(2)]
        s["V"] = [np.empty(N * n * n) for _ in range(2)]
        return s
    s["z"] = z
    s["opt"] = ves.default_options(vnorm=ves.VNORM_TWO, precision=case.get("prec", 0),
                                   want_vectors=int(kind == "solve"))
    s["A"], s["E"] = _planes(N * n * n, 2), _planes(N * n, 2)
    s["V"] = _planes(N * n * n, 2) if kind == "solve" else (None, None)
    s["ws"] = ves.Workspace(n, case["bc"], tc, options=s["opt"])
    s["Zv"], s["Ze"] = _complex_buffers(N, n)
    return s


def _complex_buffers(N, n):
    return (torch.empty(N, n, n, dtype=torch.complex128, device=DEV),
            torch.empty(N, n, dtype=torch.complex128, device=DEV))


def _ordered(E, V=None):
    """Eigenvalues ascending by real part, vectors with a real first component."""
    order = torch.argsort(E.real, dim=1)
    E = torch.gather(E, 1, order)
    if V is None:
        return E
    V = torch.gather(V, 2, order[:, None, :].expand(V.shape))
    first = V[:, :1, :]
    return E, V * (first.conj() / first.abs())


def run(s):
    kind = s["kind"]
    if kind == "varsize":
        ves.eigensolve_varsize(s["count"], s["nmax"], s["dims"], *s["A"], *s["E"], *s["V"], options=s["opt"],
                               workspace=s["ws"])
        E, V = torch.complex(*s["E"]), torch.complex(*s["V"])
        order = torch.argsort(E.real)
        order = order[torch.argsort(s["mat"][order], stable=True)]
        V = V[s["start"][order][s["col"]] + s["row"]]
        first = V[s["start"]]
        return E[order], V * (first.conj() / first.abs())[s["col"]]
    n, bc, tc, N = s["n"], s["bc"], s["tc"], s["bc"] * s["tc"]
    if kind == "host":
        for t, a in zip(s["T"], s["A"]):  # the call overwrites its input
            np.copyto(t, a)
        ves.eigensolver(n, bc, tc, *s["T"], *s["E"], *s["V"])
        E, V = (torch.complex(*(torch.from_numpy(x).to(DEV) for x in s[k])) for k in ("E", "V"))
        E = E.view(bc, n, tc).transpose(1, 2).reshape(N, n)
        V = V.view(bc, n, n, tc).permute(0, 3, 2, 1).reshape(N, n, n)
        return _ordered(E, V / torch.linalg.vector_norm(V, dim=1, keepdim=True))
    if kind == "learned":
        s["net"].predict_into(N, tc, s["p"], *s["A"], *s["S"], s["pws"])
        ves.eigensolve_shifts(n, bc, tc, *s["A"], *s["E"], *s["V"], *s["S"], options=s["opt"], workspace=s["ws"])
    else:
        ves.soa_from_complex_dev(n, bc, tc, s["z"], *s["A"])
        ves.eigensolve(n, bc, tc, *s["A"], *s["E"], *s["V"], options=s["opt"], workspace=s["ws"])
    ves.complex_from_soa_vec_dev(n, bc, tc, *s["E"], s["Ze"])
    if kind == "values":
        return _ordered(s["Ze"])
    ves.complex_from_soa_dev(n, bc, tc, *s["V"], s["Zv"])
    return _ordered(s["Ze"], s["Zv"])


def work(case):
    """A read once, eigenvalues and vectors written once; the flops of the
    reduction, of 3.3 QR sweeps per eigenvalue and of the vectors (24 n^3 +
    66 n^3; without vectors 40/3 n^3 + 22 n^3)."""
    if case["kind"] == "varsize":
        ns = np.arange(case["nmin"], case["nmax"] + 1, dtype=float)
        return {"bytes": case["count"] * float(np.mean(32 * ns ** 2 + 16 * ns)),
                "flops": case["count"] * float(np.mean(90 * ns ** 3))}
    n, N = case["n"], case["bc"] * case["tc"]
    if case["kind"] == "values":
        return {"bytes": N * (16.0 * n * n + 16 * n), "flops": N * 35.3 * n ** 3}
    return {"bytes": N * (32.0 * n * n + 16 * n), "flops": N * 90.0 * n ** 3}


def exact(case, seed):
    """The same eigenpairs from numpy.linalg.eig, where that takes a few seconds."""
    def eig(A, vectors=True):
        if not vectors:
            return np.sort_complex(np.linalg.eigvals(A))
        w, v = np.linalg.eig(A)
        o = np.argsort(w.real, axis=1)
        w, v = np.take_along_axis(w, o, 1), np.take_along_axis(v, o[:, None, :], 2)
        return w, v * (np.conj(v[:, :1]) / np.abs(v[:, :1]))

    if case["kind"] == "varsize":
        if work(case)["flops"] > 2e10:
            return None
        dims, _, _, groups = _varsize_inputs(case, seed)
        E, V = [None] * len(dims), [None] * len(dims)
        for idx, A in groups:
            w, v = eig(A.cpu().numpy())
            for k, m in enumerate(idx.tolist()):
                E[m], V[m] = w[k], v[k].T.reshape(-1)
        return np.concatenate(E), np.concatenate(V)
    n, tc, N = case["n"], case["tc"], case["bc"] * case["tc"]
    if N * 90.0 * n ** 3 > 4e10 or N > 60_000:
        return None
    if case["kind"] == "learned":
        _, re, im = learned_shift.family(N, n, param_seed=seed, thread_cnt=tc, device=DEV)
        A = torch.complex(re, im).view(-1, n, n, tc).permute(0, 3, 2, 1).reshape(N, n, n)
    else:
        A = _gauss(torch.Generator(device=DEV).manual_seed(seed), N, n, n)
    return eig(A.cpu().numpy(), case["kind"] != "values")
