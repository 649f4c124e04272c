"""The fixed-point solve's device code on the CPU, its lanes taking turns in
several orders: what a lane computes between two barriers must not depend on
which lane runs first, and lanes must meet at the same barrier."""
import numpy as np
import pytest

import fx_host

ORDERS = (0, 1, 2)  # ascending, descending, random


def batch(n, N):
    """Complex Gaussian, one Hermitian; one triangular, which the fixed-point form leaves."""
    rng = np.random.default_rng(n)
    A = rng.standard_normal((N, n, n)) + 1j * rng.standard_normal((N, n, n))
    A[1] = (A[1] + A[1].conj().T) / 2
    A[2] = np.triu(A[2])
    return A


def check_orders(A, form, vec):
    ref = fx_host.solve(A)
    assert not ref["error"] and ref["ok"][2] == 0 and (np.delete(ref["ok"], 2) == 1).all()
    for order in ORDERS:
        out = fx_host.solve(A, form, vec, order)
        assert not out["error"], (order, out["error"])
        for key in ("ok", "sweeps", "E") + (("V",) if vec else ()):
            np.testing.assert_array_equal(out[key], ref[key], err_msg="%s, order %d" % (key, order))


# a chunk of rotations and less, one more, several; windows that end inside a chunk
@pytest.mark.parametrize("n,N", [(3, 40), (8, 33), (9, 20), (16, 20), (19, 9)])
@pytest.mark.parametrize("form", ["l1", "l2", "l4", "l8"])
@pytest.mark.parametrize("vec", [True, False])
def test_lanes_in_any_order(n, N, form, vec):
    check_orders(batch(n, N), form, vec)


# several rounds of a warp's groups, with a matrix that the guard refuses in some of them and
# groups without a matrix in the last
@pytest.mark.parametrize("n,N,form", [(3, 37, "g4"), (9, 37, "g4"), (16, 21, "g4"), (9, 17, "g8"), (16, 17, "g8"),
                                      (9, 9, "g16"), (19, 9, "g16"), (9, 4, "g32"), (9, 3, "g64")])
@pytest.mark.parametrize("vec", [True, False])
def test_groups_in_any_order(n, N, form, vec):
    check_orders(batch(n, N), form, vec)


def test_solves_in_fixed_point():
    A = batch(12, 8)
    out = fx_host.solve(A)
    for k in np.nonzero(out["ok"])[0]:
        R = A[k] @ out["V"][k] - out["V"][k] * out["E"][k]
        assert np.linalg.norm(R, axis=0).max() <= 1e-14 * np.linalg.norm(A[k])
