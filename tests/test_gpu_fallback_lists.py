"""The FP32+refine form's fallback list: kernels chosen by its length, which only
the device knows, and what a short one in a large batch costs."""
import numpy as np
import pytest

import ves
from test_gpu_mixed import run_fused_opts

pytestmark = pytest.mark.gpu
MIX = ves.VES_PREC_FP32_REFINE


def batch_on_device(n, N, big):
    """Gaussian matrices, the first `big` of them beyond FP32's range: they fall back."""
    import torch
    g = torch.Generator(device="cuda").manual_seed(n)
    planes = [torch.randn(n * n, N, generator=g, dtype=torch.float64, device="cuda") for _ in range(2)]
    for p in planes:
        p[:, :big] *= 1e30
    E = [torch.empty(N * n, dtype=torch.float64, device="cuda") for _ in range(2)]
    V = [torch.empty(N * n * n, dtype=torch.float64, device="cuda") for _ in range(2)]
    return [p.view(-1) for p in planes], E, V, torch.empty(N, dtype=torch.int32, device="cuda")


# lists shorter and longer than what the group kernel takes
@pytest.mark.parametrize("n,N,big", [(9, 60000, 300), (9, 60000, 40000), (16, 60000, 2000), (16, 60000, 30000),
                                     (32, 20000, 500), (32, 20000, 12000), (48, 6000, 5), (48, 6000, 5000)])
def test_short_and_long_fallback_lists_same_bits(n, N, big):
    import torch
    A, E, V, st = batch_on_device(n, N, big)
    ves.eigensolve(n, 1, N, *A, *E, *V, status=st)
    torch.cuda.synchronize()
    want = [x.view(-1, N)[:, :big].cpu().numpy() for x in E + V]
    ves.eigensolve(n, 1, N, *A, *E, *V, status=st, options=ves.default_options(precision=MIX))
    torch.cuda.synchronize()
    fell = (st.cpu().numpy() & ves.VES_STATUS_REFINE_FALLBACK) != 0
    assert fell[:big].all() and fell.sum() <= big + 3
    for got, ref in zip(E + V, want):
        np.testing.assert_array_equal(got.view(-1, N)[:, :big].cpu().numpy(), ref)


@pytest.mark.parametrize("n,N", [(24, 131072), (32, 65536)])
def test_one_fallback_matrix_costs_little(n, N):
    """One matrix that falls back in a full batch: a quarter of the batch's time at
    most (one lane of the lane kernel takes 0.3 and 0.8 of it)."""
    import torch
    times = []
    for big in (0, 1):
        A, E, V, st = batch_on_device(n, N, big)
        opt = ves.default_options(precision=MIX)
        ws = ves.Workspace(n, 1, N, options=opt)
        t = []
        for _ in range(4):
            a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            a.record()
            ves.eigensolve(n, 1, N, *A, *E, *V, status=st, options=opt, workspace=ws)
            b.record()
            torch.cuda.synchronize()
            t.append(a.elapsed_time(b))
        times.append(min(t[1:]))
    assert times[1] <= 1.25 * times[0], times


def test_forced_fallback_of_a_whole_batch():
    """Every matrix on the list, more of them than a launch of the group kernel takes."""
    rng = np.random.default_rng(31)
    A = rng.standard_normal((9000, 12, 12)) + 1j * rng.standard_normal((9000, 12, 12))
    ref = run_fused_opts(A, 3000)
    out = run_fused_opts(A, 3000, precision=MIX, refine_steps=0)
    for key in ("E", "V", "sweeps"):
        np.testing.assert_array_equal(out[key], ref[key])
