"""Batches in which the fixed-point form leaves matrices to the FP64 kernels:
results, and that the forms with many matrices per warp keep them apart."""
import numpy as np
import pytest

import oracle
import ves
from gpu_util import dev, run_fused
from parity import match_eigs, residuals
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


# lengths on both sides of the one at which a list goes from a matrix per warp (two rows and
# columns per lane for n > 32) to one per lane
@pytest.mark.parametrize("n,N", [(3, 2600), (10, 5000), (24, 4400), (32, 3800), (40, 2600), (64, 1900)])
def test_fp64_list_kernels_same_bits(n, N):
    rng = np.random.default_rng(1000 + n)
    A = cgauss(rng, (N, n, n))
    A[:, n // 2:, :n // 2] = 0
    A[3] = np.triu(A[3])  # the reflectors' trivial branch
    long_list = run_fused(A, N, want_T=True, vnorm=1)
    assert (long_list["status"] == 0).all()
    for s in (0, N - 60):
        short = run_fused(A[s:s + 60], 60, want_T=True, vnorm=1)
        for key, want in short.items():
            assert np.array_equal(long_list[key][s:s + 60], want), key
    # (the oracle, like the reference, divides by a subdiagonal that is exactly zero)
    _, err, _ = match_eigs(long_list["E"][:60], np.linalg.eigvals(A[:60]))
    assert (err / np.linalg.norm(A[:60], axis=(1, 2))).max() <= 1e-12


# orders whose Newton step keeps its scratch beside the slot, not in Z, and the next one
@pytest.mark.parametrize("n", [2, 3, 4, 5, 6])
@pytest.mark.parametrize("polish", [0, 4])
def test_shifts_of_small_orders(n, polish, monkeypatch):
    import torch
    monkeypatch.setenv("VES_POLISH_FP64_STEP", "2")
    rng = np.random.default_rng(1100 + n)
    N, tc = 96, 8
    A = cgauss(rng, (N, n, n))
    A[::9, n // 2:, :n // 2] = 0  # solved in FP64
    ref = np.linalg.eigvals(A)
    planes = [dev(x) for x in ves.soa_from_complex(A, tc)]
    S = [dev(x) for x in ves.soa_vec_from_complex(ref + 1e-3 * cgauss(rng, ref.shape), tc)]
    E = [torch.empty(N * n, dtype=torch.float64, device="cuda") for _ in range(2)]
    V = [torch.empty_like(planes[0]) for _ in range(2)]
    st = torch.full((N,), -1, dtype=torch.int32, device="cuda")
    ves.eigensolve_shifts(n, N // tc, tc, *planes, *E, *V, *S, status=st, options=ves.default_options(shift_polish=polish))
    torch.cuda.synchronize()
    got = ves.complex_vec_from_soa(E[0].cpu().numpy(), E[1].cpu().numpy(), n, tc)
    vec = ves.complex_from_soa(V[0].cpu().numpy(), V[1].cpu().numpy(), n, tc)
    assert ((st.cpu().numpy() & ~ves.VES_STATUS_SHIFT_FALLBACK) == 0).all()
    _, err, _ = match_eigs(got, ref)
    assert (err / np.linalg.norm(A, axis=(1, 2))).max() <= 1e-12
    assert residuals(A, got, vec).max() <= 1e-13


def test_noalloc_beyond_one_slice():
    """More matrices than the allocation-free call lists at once (2^20): the slices after the
    first start inside the batch; refused matrices in each."""
    import ctypes
    import torch
    n, N = 3, (1 << 20) + 37
    g = torch.Generator(device="cuda").manual_seed(3)
    A = [torch.randn(n, n, N, generator=g, dtype=torch.float64, device="cuda") for _ in range(2)]  # [column][row][matrix]
    for p in A:
        p[0, 1:, ::5] = 0  # first column: reducible
        p[0, 1:, N - 1] = 0
    planes = [p.view(-1) for p in A]
    outs = []
    for noalloc in (False, True):
        o = [torch.full((k,), float("nan"), dtype=torch.float64, device="cuda") for k in (N * n, N * n, N * n * n, N * n * n)]
        st = torch.full((N,), -1, dtype=torch.int32, device="cuda")
        if noalloc:
            ptr = [ctypes.c_void_p(t.data_ptr()) for t in planes + o + [st]]
            stream = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
            assert ves.lib().ves_eigensolve_noalloc(n, 1, N, *ptr, stream) == 0, ves.last_error()
        else:
            ves.eigensolve(n, 1, N, *planes, *o, status=st)
        torch.cuda.synchronize()
        assert int(st.abs().max()) == 0
        outs.append(o)
    for a, b in zip(*outs):
        assert torch.equal(a, b)
