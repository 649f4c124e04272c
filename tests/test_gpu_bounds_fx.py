"""The bounds-checked build on every form of the fixed-point solve, the warp
Schur kernel with two rows per lane and the refinement by matrix: the checks of
their pointer loops and shared-memory layouts count nothing, and the results
meet the residual bar.  In a child process bound to the checked library."""
import os
import subprocess
import sys

import pytest

from test_gpu_bounds import CHILD, PKG

pytestmark = pytest.mark.gpu

# the helpers of the other bounds test, then other calls
BODY = CHILD[:CHILD.index("rng = np.random.default_rng(5)")] + r'''
rng = np.random.default_rng(6)
smem = lambda n, G, vec: max(32 // G, 1) * ((2 if vec else 1) * n * (n + 1) + 2 * n) * 16
for n in (3, 4, 9, 16, 17, 33, 64):
    A = cg(rng, (45, n, n))
    A[::5, n // 2:, :n // 2] = 0                                    # left to the FP64 kernels
    for form in ("l1", "l2", "l4", "l8", "g4", "g8", "g16", "g32", "g64", "g128"):
        G = int(form[1:])
        if form[0] == "g" and (G > (4 if G <= 32 else 2) * n or smem(n, G, True) > 220000):
            continue
        os.environ["VES_FX_LANES"] = form
        solve(A, 9, schur=True)
        solve(A, 9, want_vectors=0)
os.environ.pop("VES_FX_LANES")
for n in (3, 8, 15, 16, 24, 33, 41, 64):
    solve(cg(rng, (45, n, n)), 9, precision=1)                      # Schur kernels by warp, refinement by matrix
    solve(cg(rng, (45, n, n)), 9, precision=1, refine_steps=0)      # fallback lists
# mixed sizes: a few large among small ones (eight lanes per matrix) and the other way round
for sizes in ([64] * 3 + [41] * 2 + [9] * 70, [3, 4, 5] * 20 + [12]):
    sizes = np.array(sizes)
    mats = [cg(rng, (k, k)) for k in sizes]
    flat = np.concatenate([m.T.reshape(-1) for m in mats])
    o = [torch.empty(int(sizes.sum()), dtype=torch.float64, device="cuda") for _ in range(2)] + \
        [torch.empty(flat.size, dtype=torch.float64, device="cuda") for _ in range(2)]
    ves.eigensolve_varsize(len(sizes), int(sizes.max()), dev(sizes.astype(np.int32)), dev(flat.real.copy()),
                           dev(flat.imag.copy()), *o)
# learned shifts of small orders (their scratch is not in Z), with polish and the FP64 step
for n in (2, 3, 4, 5, 6):
    A = cg(rng, (40, n, n))
    planes = [dev(x) for x in ves.soa_from_complex(A, 8)]
    S = [dev(x) for x in ves.soa_vec_from_complex(np.linalg.eigvals(A), 8)]
    o = [torch.empty(40 * n, dtype=torch.float64, device="cuda") for _ in range(2)] + \
        [torch.empty(40 * n * n, dtype=torch.float64, device="cuda") for _ in range(2)]
    ves.eigensolve_shifts(n, 5, 8, *planes, *o, *S, options=ves.default_options(shift_polish=4))
torch.cuda.synchronize()
cnt = ctypes.c_ulonglong(99)
assert ves.lib().ves_bounds_violations(ctypes.byref(cnt), 1) == 0
print("VIOLATIONS", cnt.value)
'''


def test_bounds_checked_fixed_point_forms():
    import build as ves_build
    lib = ves_build.build(variant="bc")
    env = dict(os.environ, VES_LIBRARY=lib, VES_PKG=PKG, VES_AUTOBUILD="0")
    r = subprocess.run([sys.executable, "-c", BODY], env=env, capture_output=True, text=True, timeout=900)
    assert r.returncode == 0, r.stdout[-3000:] + r.stderr[-3000:]
    line = [ln for ln in r.stdout.splitlines() if ln.startswith("VIOLATIONS")]
    assert line and line[0].split()[1] == "0", r.stdout[-2000:]
