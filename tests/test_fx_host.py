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


def bordered(rng, N, n, eps, hermitian, first=0):
    """A weak block (entries of size eps) beside strong rows and columns: row and column
    `first`, and before it a chain of couplings, so that no reflector mixes the two."""
    A = eps * (rng.standard_normal((N, n, n)) + 1j * rng.standard_normal((N, n, n)))
    strong = rng.standard_normal((N, n, n)) + 1j * rng.standard_normal((N, n, n))
    A[:, first, first:], A[:, first:, first] = strong[:, first, first:], strong[:, first:, first]
    A[:, :first, :], A[:, :, :first] = 0, 0
    for k in range(first):
        A[:, k, k:k + 2], A[:, k:k + 2, k] = strong[:, k, k:k + 2], strong[:, k:k + 2, k]
    return (A + A.conj().transpose(0, 2, 1)) / 2 if hermitian else A


@pytest.mark.parametrize("n,first", [(3, 0), (4, 0), (5, 1), (8, 0), (8, 2), (13, 5), (16, 0), (33, 0)])
@pytest.mark.parametrize("hermitian", [False, True])
@pytest.mark.parametrize("form", ["l1", "l4", "g8"])
def test_weak_block_is_left_to_fp64(n, first, hermitian, form):
    rng = np.random.default_rng(50 + n)
    A = np.concatenate([bordered(rng, 1, n, 2.0 ** -k, hermitian, first) for k in range(9, 28)])
    out = fx_host.solve(A, form)
    assert not out["error"] and not out["ok"].any()


@pytest.mark.parametrize("n", [3, 4, 5, 8, 16, 33, 64])
def test_ordinary_matrices_stay_in_fixed_point(n):
    rng = np.random.default_rng(60 + n)
    N = 200 if n <= 16 else 12
    A = rng.standard_normal((N, n, n)) + 1j * rng.standard_normal((N, n, n))
    H = (A + A.conj().transpose(0, 2, 1)) / 2
    phase = np.exp(2j * np.pi * rng.random((N, n, n)))
    chain = np.zeros((1, n, n), complex)
    chain[0] = np.diag(rng.uniform(-1, 1, n)) + np.diag(np.ones(n - 1), 1) + np.diag(np.ones(n - 1), -1)
    for B in (A, H, A.real + 0j, phase, bordered(rng, N, n, 1 / 4, False), chain):
        assert fx_host.solve(B)["ok"].all()


@pytest.mark.parametrize("n", [3, 5, 16, 33, 64])
@pytest.mark.parametrize("form", ["l1", "l2", "g8"])
def test_matrices_not_connected_from_the_first_index(n, form):
    """Diagonal, triangular and block-triangular matrices are refused; those whose nonzeros
    lead from index 1 to all others, in one step or in n - 1, are not."""
    rng = np.random.default_rng(70 + n)
    A = rng.standard_normal((1, n, n)) + 1j * rng.standard_normal((1, n, n))
    p = n // 2
    refused = [A * np.eye(n), np.triu(A), A.copy(), A.copy()]
    refused[2][:, p:, :p] = 0
    refused[3][:, n - 1, :n - 1] = 0
    out = fx_host.solve(np.concatenate(refused), form)
    assert not out["error"] and not out["ok"].any()
    cycle = np.zeros((1, n, n), complex)
    cycle[0, np.arange(n), (np.arange(n) + 1) % n] = 1  # the last index is reached first
    chain = np.triu(np.tril(A, 1), -1)
    arrow = A * ((np.arange(n)[:, None] == 0) | (np.arange(n) == 0) | np.eye(n, dtype=bool))
    out = fx_host.solve(np.concatenate([A, A.conj().transpose(0, 2, 1), chain, cycle + 0.1 * np.eye(n), arrow]), form)
    assert not out["error"]
    assert out["ok"].all()
