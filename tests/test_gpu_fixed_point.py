"""The fixed-point form of the FP64 solve, its lanes-per-matrix kernels and its
guard, and the FP32+refine kernels that hold a matrix per group of lanes or per
block, at the sizes where a tile, a warp or a range ends.

Tolerances are the solver's: eigenvalues within 1e-12 ||A||_F, residuals
||A v - lambda v|| / (||A||_F ||v||) at most 1e-13.  Kernels that differ only in
how many lanes share a matrix give the same bits (sums of products are exact
before they are rounded, every other step is done alike)."""
import numpy as np
import pytest

import ves
from gpu_util import dev, run_fused
from parity import match_eigs, residuals

pytestmark = pytest.mark.gpu
MIX = ves.VES_PREC_FP32_REFINE


def cgauss(rng, shape):
    return rng.standard_normal(shape) + 1j * rng.standard_normal(shape)


def check(A, out, scale=None):
    nA = np.linalg.norm(A, axis=(1, 2)) if scale is None else scale
    _, err, _ = match_eigs(out["E"], np.linalg.eigvals(A))
    assert (err / nA).max() <= 1e-12, (err / nA).max()
    assert residuals(A, out["E"], out["V"]).max() <= 1e-13


def forms(n):
    """The lane kernels and the group kernels that a batch of this order can take
    (a warp's matrices have to fit the shared memory of an SM)."""
    return ["l2", "l4", "l8"] + ["g%d" % G for G in (4, 8, 16, 32, 64, 128)
                                 if G <= (4 * n if G <= 32 else 2 * n)
                                 and max(32 // G, 1) * (2 * n * (n + 2) + 2 * n) * 16 <= 224 * 1024]


# N leaves the last warp of every kernel partly empty; tc = 1, odd, and N
@pytest.mark.parametrize("n,N,tc", [(3, 45, 5), (4, 33, 1), (9, 51, 51), (16, 70, 7), (17, 37, 37), (33, 21, 3),
                                    (64, 11, 11)])
def test_lanes_per_matrix_same_bits(n, N, tc, monkeypatch):
    rng = np.random.default_rng(100 + n)
    A = cgauss(rng, (N, n, n))
    A[1] = (A[1] + A[1].conj().T) / 2
    A[2] = np.triu(A[2])  # left to the FP64 kernels
    monkeypatch.setenv("VES_FX_LANES", "l1")
    ref = run_fused(A, tc, want_T=True, vnorm=2)
    check(A, ref)
    assert (ref["status"] == 0).all()
    for form in forms(n):
        monkeypatch.setenv("VES_FX_LANES", form)
        out = run_fused(A, tc, want_T=True, vnorm=2)
        for key, want in ref.items():
            assert np.array_equal(out[key], want), (form, key)


@pytest.mark.parametrize("n,N,tc", [(3, 45, 5), (16, 70, 7), (33, 21, 3), (64, 11, 11)])
def test_values_only_same_bits(n, N, tc, monkeypatch):
    import torch
    A = cgauss(np.random.default_rng(200 + n), (N, n, n))
    planes = [dev(x) for x in ves.soa_from_complex(A, tc)]
    for form in ["l1"] + forms(n):
        monkeypatch.setenv("VES_FX_LANES", form)
        E = [torch.empty(N * n, dtype=torch.float64, device="cuda") for _ in range(2)]
        ves.eigensolve(n, N // tc, tc, *planes, *E, None, None, options=ves.default_options(want_vectors=0))
        got = ves.complex_vec_from_soa(E[0].cpu().numpy(), E[1].cpu().numpy(), n, tc)
        assert np.array_equal(got, run_fused(A, tc)["E"]), form


@pytest.mark.parametrize("n", [3, 16, 40])
def test_guard_keeps_relative_accuracy(n):
    """One scale per matrix does not serve matrices whose blocks differ widely
    in size, that are reducible, zero or of an extreme exponent: they keep the
    accuracy of the FP64 kernels (eigenvalues of a small block to 1e-12 of that
    block), beside ordinary matrices in the same batch."""
    rng = np.random.default_rng(300 + n)
    N, tc = 24, 8
    A = cgauss(rng, (N, n, n))
    p = n // 2
    for k, s in ((1, 1e-6), (2, 1e-12), (3, 1e-30)):
        A[k] = 0
        A[k, :p, :p] = cgauss(rng, (p, p))
        A[k, p:, p:] = s * cgauss(rng, (n - p, n - p))
    A[4] = 0
    A[5] = np.triu(A[5])
    A[6] = np.diag(np.diag(A[6]))
    A[7] *= 1e-290
    A[8] *= 1e150
    A[9] *= 1e-150
    out = run_fused(A, tc)
    # (squares of 1e-290 underflow in the FP64 kernels: the iteration cap reports it)
    ok = np.arange(N) != 7
    assert out["status"][7] & 1 and (out["status"][ok] == 0).all()
    A, out = A[ok], {key: v[ok] for key, v in out.items()}
    scale = np.maximum(np.linalg.norm(A, axis=(1, 2)), 1e-300)
    _, err, _ = match_eigs(out["E"], np.linalg.eigvals(A))
    assert (err / scale).max() <= 1e-12
    nv = np.linalg.norm(out["V"], axis=1)
    R = (A / scale[:, None, None]) @ out["V"] - out["V"] * (out["E"] / scale[:, None])[:, None, :]
    assert (np.linalg.norm(R, axis=1) / nv).max() <= 1e-13
    for k, s in ((1, 1e-6), (2, 1e-12), (3, 1e-30)):
        small = np.linalg.eigvals(A[k, p:, p:])
        got = out["E"][k][np.argsort(np.abs(out["E"][k]))[:n - p]]
        _, e, _ = match_eigs(got[None], small[None])
        assert e[0] <= 1e-12 * np.linalg.norm(A[k, p:, p:]), (s, e[0])


def test_guard_nonfinite_flagged():
    rng = np.random.default_rng(7)
    A = cgauss(rng, (40, 12, 12))
    A[3, 2, 5] = np.nan
    A[17, 0, 0] = np.inf
    out = run_fused(A, 8)
    ok = np.ones(40, bool)
    ok[[3, 17]] = False
    assert (out["status"][ok] == 0).all() and (out["status"][~ok] != 0).all()
    check(A[ok], {k: v[ok] for k, v in out.items()})


# orders at the edges of the refinement's tiles (4 to 16 rows, 8 columns) and warps
# per block, and of the warp Schur kernel's one and two rows per lane
@pytest.mark.parametrize("n", [1, 3, 4, 5, 8, 9, 12, 13, 15, 16, 17, 23, 24, 25, 28, 29, 31, 32, 33, 40, 41, 48, 49, 56,
                               57, 63, 64])
@pytest.mark.parametrize("vnorm", [0, 1, 2])
def test_mixed_small_batches(n, vnorm):
    rng = np.random.default_rng(400 + n)
    N, tc = 35, (1, 7, 35)[vnorm]
    A = cgauss(rng, (N, n, n))
    A[:10] = (A[:10] + A[:10].conj().transpose(0, 2, 1)) / 2
    A[10:13] *= np.array([1e-16, 1e-8, 1e16])[:, None, None]
    out = run_fused(A, tc, precision=MIX, vnorm=vnorm)
    check(A, out)
    assert (out["status"] & ~ves.VES_STATUS_REFINE_FALLBACK == 0).all()
    assert ((out["status"] & ves.VES_STATUS_REFINE_FALLBACK) != 0).mean() <= 0.2
    size = np.linalg.norm(out["V"], axis=1) if vnorm == 2 else (np.abs(out["V"].real) + np.abs(out["V"].imag)).max(1)
    if vnorm:
        assert np.abs(size - 1).max() <= 1e-14


@pytest.mark.parametrize("n,N,tc", [(9, 4097, 4097), (12, 4100, 100), (15, 4101, 3), (16, 16389, 9), (16, 4099, 4099),
                                    (24, 4104, 8), (27, 4100, 4), (32, 4096, 512)])
def test_mixed_larger_batches(n, N, tc):
    """Across the batch sizes and orders at which the Schur and refinement kernels change."""
    A = cgauss(np.random.default_rng(500 + n), (N, n, n))
    out = run_fused(A, tc, precision=MIX)
    assert residuals(A, out["E"], out["V"]).max() <= 1e-13
    check(A[-40:], {k: v[-40:] for k, v in out.items()})
    assert (out["status"] & ~ves.VES_STATUS_REFINE_FALLBACK == 0).all()


@pytest.mark.parametrize("count", [(3, 40), (33, 500)])
def test_varsize_few_large_among_many_small(count):
    """Orders whose one-lane work would outlast the batch get eight lanes per
    matrix: same bits as the fixed-size solver."""
    import torch
    rng = np.random.default_rng(600)
    dims = np.concatenate([np.full(count[0], 64), np.full(count[0] + 2, 41), np.full(count[1], 10), [3, 4, 63]])
    dims = rng.permutation(dims).astype(np.int32)
    mats = [cgauss(rng, (d, d)) for d in dims]
    flat = np.concatenate([M.T.ravel() for M in mats])
    A = [dev(x) for x in (flat.real.copy(), flat.imag.copy())]
    E = [torch.empty(int(dims.sum()), dtype=torch.float64, device="cuda") for _ in range(2)]
    V = [torch.empty_like(A[0]) for _ in range(2)]
    opt = ves.default_options()
    ves.eigensolve_varsize(len(dims), 64, dev(dims), *A, *E, *V, options=opt,
                           workspace=ves.varsize_workspace(len(dims), 64, opt))
    torch.cuda.synchronize()
    gotE, gotV = (p[0].cpu().numpy() + 1j * p[1].cpu().numpy() for p in (E, V))
    eo, vo = np.cumsum(dims) - dims, np.cumsum(dims.astype(np.int64) ** 2) - dims.astype(np.int64) ** 2
    for d in np.unique(dims):
        idx = np.nonzero(dims == d)[0]
        ref = run_fused(np.stack([mats[i] for i in idx]), 1)
        for k, i in enumerate(idx):
            assert np.array_equal(gotE[eo[i]:eo[i] + d], ref["E"][k]), (d, i)
            assert np.array_equal(gotV[vo[i]:vo[i] + d * d].reshape(d, d).T, ref["V"][k]), (d, i)


@pytest.mark.parametrize("n,N", [(8, 5000), (16, 9000)])
def test_long_and_short_fp64_lists_same_bits(n, N):
    """A batch that the fixed-point form leaves to FP64 altogether: a long list
    goes one matrix per lane, short ones one per warp, with the same bits."""
    rng = np.random.default_rng(700 + n)
    A = cgauss(rng, (N, n, n))
    A[:, n // 2:, :n // 2] = 0
    out = run_fused(A, N, vnorm=2)
    check(A[:40], {k: v[:40] for k, v in out.items()})
    for s in (0, N - 100):
        part = run_fused(A[s:s + 100], 100, vnorm=2)
        for key, want in part.items():
            assert np.array_equal(out[key][s:s + 100], want), key
