"""Batches in which the fixed-point form leaves matrices to the FP64 kernels:
results, and that the forms with many matrices per warp keep them apart."""
import numpy as np
import pytest

from gpu_util import run_fused

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
