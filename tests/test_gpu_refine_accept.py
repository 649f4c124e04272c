"""What the FP32+refine form accepts: ||A v - lambda v|| <= refine_tol ||A||_F ||v||
of the pairs as returned, in extended precision."""
import numpy as np
import pytest

import ves
import workloads

pytestmark = pytest.mark.gpu
MIX = ves.VES_PREC_FP32_REFINE


# Full batches, so that the largest of millions of accepted residuals lies at the limit (the
# first: the benchmark's).  The limit is strict: the form's own margin, six standard deviations
# of its residual's rounding, covers that of the returned vector (0.05% of the limit) as well.
@pytest.mark.parametrize("n,N,seed", [(16, 1 << 20, None), (16, 1 << 20, 1), (32, 1 << 16, 0), (57, 1 << 12, 0)])
def test_accepted_residuals_within_tolerance(n, N, seed):
    import torch
    if seed is None:
        A = [torch.from_numpy(x).cuda().view(N // 512, n, n, 512).permute(1, 2, 0, 3).reshape(n, n, N).contiguous()
             for x in workloads.gaussian_soa(N, n, 1, 512)]
    else:
        g = torch.Generator(device="cuda").manual_seed(seed)
        A = [torch.randn(n, n, N, generator=g, dtype=torch.float64, device="cuda") for _ in range(2)]  # [column][row][matrix]
    E = [torch.empty(n, N, dtype=torch.float64, device="cuda") for _ in range(2)]
    V = [torch.empty(n, n, N, dtype=torch.float64, device="cuda") for _ in range(2)]
    opt = ves.default_options(precision=MIX)
    ves.eigensolve(n, 1, N, *(x.view(-1) for x in A + E + V), options=opt)
    nA = (A[0] ** 2 + A[1] ** 2).sum((0, 1)).sqrt()
    res = torch.empty(n, N, dtype=torch.float64, device="cuda")
    for k in range(n):  # pair k: A v_k - lambda_k v_k, rows along dimension 0
        vr, vi, er, ei = V[0][k], V[1][k], E[0][k], E[1][k]
        rr, ri = vi * ei - vr * er, -(vr * ei + vi * er)
        for j in range(n):
            rr += A[0][j] * vr[j] - A[1][j] * vi[j]
            ri += A[0][j] * vi[j] + A[1][j] * vr[j]
        res[k] = ((rr ** 2 + ri ** 2).sum(0) / (vr ** 2 + vi ** 2).sum(0)).sqrt() / nA
    top = torch.topk(res.view(-1), 40).indices.cpu().numpy()
    worst = 0.0
    for k, m in zip(top // N, top % N):
        a, v = ((x[0][..., m] + 1j * x[1][..., m]).cpu().numpy().astype(np.clongdouble) for x in (A, (V[0][k], V[1][k])))
        lam = np.clongdouble(E[0][k, m].item()) + 1j * np.clongdouble(E[1][k, m].item())
        r = (a * v[:, None]).sum(0) - lam * v
        size = lambda x: np.sqrt((x.real ** 2 + x.imag ** 2).sum())  # noqa: E731
        worst = max(worst, float(size(r) / (size(a) * size(v))))
    assert worst <= opt.refine_tol, worst
