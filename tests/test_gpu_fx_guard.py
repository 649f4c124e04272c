"""Batches in which the fixed-point form leaves matrices to the FP64 kernels:
results, and that the forms with many matrices per warp keep them apart."""
import numpy as np
import pytest

import oracle
import ves
from gpu_util import dev, run_fused
from parity import match_eigs
from test_fx_host import bordered

pytestmark = pytest.mark.gpu


def cgauss(rng, shape):
    return rng.standard_normal(shape) + 1j * rng.standard_normal(shape)


# several rounds of every warp of the GPU (152 SMs, at most 21 blocks of 32 / G matrices on each)
@pytest.mark.parametrize("n,N,form", [(9, 60007, "g4"), (16, 30011, "g8"), (16, 15013, "g16"), (16, 30011, "l2"),
                                      (16, 30011, "l8")])
def test_guarded_matrices_among_rounds_same_bits(n, N, form, monkeypatch):
    rng = np.random.default_rng(800 + n)
    A = cgauss(rng, (N, n, n))
    A[::7, n // 2:, :n // 2] = 0  # block triangular: left to the FP64 kernels
    A[5::11] = np.triu(A[5::11])
    monkeypatch.setenv("VES_FX_LANES", "l1")
    ref = run_fused(A, N, vnorm=2)
    assert (ref["status"] == 0).all()
    monkeypatch.setenv("VES_FX_LANES", form)
    out = run_fused(A, N, vnorm=2)
    for key, want in ref.items():
        assert np.array_equal(out[key], want), key


def small_eigs(E, count):
    return np.take_along_axis(E, np.argsort(np.abs(E), axis=1)[:, :count], axis=1)


def weak_block_batch(n, first):
    """A weak block of n - 1 - first rows of size 2^-k, k = 8 .. 27, beside strong rows and
    columns: the matrices, the block's norms, and its eigenvalues by the FP64 oracle (whose
    reflectors do not mix the block with the strong entries: they are good to 2^-53 of it)."""
    rng = np.random.default_rng(900 + n + first)
    A = np.concatenate([bordered(rng, 1, n, 2.0 ** -(k // 2), k % 2 == 1, first) for k in range(16, 56)])
    rA, iA = ves.soa_from_complex(A, 8)
    rE, iE, *_ = oracle.eigensolve(rA, iA, n, 8)
    count = n - 2 - first
    return A, np.linalg.norm(A[:, first + 1:, first + 1:], axis=(1, 2)), small_eigs(ves.complex_vec_from_soa(rE, iE, n, 8), count)


def check_small(E, norms, want):
    _, err, _ = match_eigs(small_eigs(E, want.shape[1]), want)
    assert (err / norms).max() <= 1e-12, (err / norms).max()


@pytest.mark.parametrize("n,first", [(3, 0), (8, 0), (8, 2), (16, 0), (40, 0)])
def test_weak_block_beside_strong_row_keeps_relative_accuracy(n, first):
    """The small eigenvalues to 1e-12 of the block, through every form of the FP64 solve."""
    import torch
    A, norms, want = weak_block_batch(n, first)
    N = len(A)
    check_small(run_fused(A, 8)["E"], norms, want)
    check_small(run_fused(A, 8, precision=ves.VES_PREC_FP32_REFINE, refine_steps=0)["E"], norms, want)
    planes = [dev(x) for x in ves.soa_from_complex(A, 8)]
    E = [torch.empty(N * n, dtype=torch.float64, device="cuda") for _ in range(2)]
    V = [torch.empty_like(planes[0]) for _ in range(2)]

    def values():
        return ves.complex_vec_from_soa(E[0].cpu().numpy(), E[1].cpu().numpy(), n, 8)
    ves.eigensolve(n, N // 8, 8, *planes, *E, None, None, options=ves.default_options(want_vectors=0))
    check_small(values(), norms, want)
    S = [dev(x) for x in ves.soa_vec_from_complex(np.linalg.eigvals(A), 8)]
    ves.eigensolve_shifts(n, N // 8, 8, *planes, *E, *V, *S, options=ves.default_options())
    check_small(values(), norms, want)
    flat = A.transpose(0, 2, 1).ravel()
    ves.eigensolve_varsize(N, n, dev(np.full(N, n, np.int32)), dev(flat.real.copy()), dev(flat.imag.copy()), *E, *V)
    check_small((E[0].cpu().numpy() + 1j * E[1].cpu().numpy()).reshape(N, n), norms, want)
