"""The data-flow Cholesky factorization, its forward and backward solves and its
explicit inverse, through solveSaddleFromA: orders at the edges of its 64 x 64
tiles (one block, a ragged last block, odd orders whose rows start on 8-byte
boundaries), right-hand sides at the edges of their groups of 16 and 64 (3 per
constraint row), and the explicit inverses of more than 64 rows.

Against numpy's LU of the whole saddle matrix. The systems are conditioned below
1e4, so both sides are within about 1e4 * n * 2^-53 = 1e-9 of the solution at the
largest order; the residual bound is the reference's."""
from __future__ import annotations

import numpy as np
import pytest

from repulsive_test2_b200 import api as T

pytestmark = pytest.mark.gpu


def _system(n, k, seed):
    rng = np.random.default_rng(seed)
    M = rng.standard_normal((n, n))
    # positive semi-definite with the constants as its kernel, as every Gram matrix of a curve
    P = np.eye(n) - np.ones((n, n)) / n
    A = P @ (M @ M.T / n + 0.5 * np.eye(n)) @ P
    A = 0.5 * (A + A.T)
    C = rng.standard_normal((k, 3 * n)) / np.sqrt(3 * n)
    return A, C, rng.standard_normal(3 * n), rng.standard_normal(k)


def _check(n, k, seed):
    A, C, b, d = _system(n, k, seed)
    K = np.zeros((3 * n + k, 3 * n + k))
    for c in range(3):
        K[c * n:(c + 1) * n, c * n:(c + 1) * n] = A
    K[3 * n:, :3 * n], K[:3 * n, 3 * n:] = C, C.T
    ref = np.linalg.solve(K, np.concatenate([b, d]))
    r = T.solveSaddleFromA(A, n, C, b, d)
    assert r["residual"] <= 1e-10
    assert np.linalg.norm(r["x"] - ref[:3 * n]) <= 1e-9 * np.linalg.norm(ref[:3 * n])
    assert np.linalg.norm(r["lambda"] - ref[3 * n:]) <= 1e-9 * max(1.0, np.linalg.norm(ref[3 * n:]))


@pytest.mark.parametrize("n", [2, 63, 64, 65, 127, 128, 129, 193, 450, 641])
def test_orders(n):
    _check(n, 4, n)


@pytest.mark.parametrize("k", [5, 6, 20, 21, 22, 43, 64])
def test_right_hand_sides(k):
    """3 (k + 1) right-hand sides: 18 .. 195 of them."""
    _check(131, k, k)


@pytest.mark.parametrize("n,k", [(96, 65), (129, 130), (200, 128), (131, 191)])
def test_explicit_inverses(n, k):
    _check(n, k, n + k)


@pytest.mark.parametrize("n,bad", [(40, 39), (200, 70), (200, 199)])
def test_breakdown(n, bad):
    """An indefinite matrix: singular, whichever block holds the pivot."""
    A, C, b, d = _system(n, 3, 1)
    A[bad, bad] -= 50.0
    with pytest.raises(T.SingularSystemError):
        T.solveSaddleFromA(A, n, C, b, d)


def test_repeats_bit_for_bit():
    """Tiles are taken in whatever order the blocks run: the result may not depend on it."""
    A, C, b, d = _system(777, 4, 3)
    first = T.solveSaddleFromA(A, 777, C, b, d)
    for _ in range(4):
        again = T.solveSaddleFromA(A, 777, C, b, d)
        assert np.array_equal(first["x"], again["x"])
        assert np.array_equal(first["lambda"], again["lambda"])


def test_rows_of_every_form():
    """More than 64 rows of all kinds: one vertex, a difference of two (also along one
    axis only), two vertices that are no difference, one vertex shared by 40 rows, and
    two dense rows."""
    n = 150
    A, _, b, _ = _system(n, 1, 5)
    rng = np.random.default_rng(6)
    C = []
    for s in range(60):
        row = np.zeros((3, n))
        w = rng.standard_normal(3) if s % 3 else np.array([0.0, 1.5, 0.0])
        p, q = (0, 1 + s) if s < 40 else (2 * s - 20, 2 * s - 19)
        row[:, p] += w
        row[:, q] -= w
        C.append(row)
    for v in (100, 105):
        for c in range(3):
            row = np.zeros((3, n))
            row[c, v] = 1.0
            C.append(row)
    for v in (110, 120, 130):
        row = np.zeros((3, n))
        row[:, v], row[:, v + 3] = rng.standard_normal(3), rng.standard_normal(3)
        C.append(row)
    C += [rng.standard_normal((3, n)) / n for _ in range(2)]
    C = np.array(C).reshape(len(C), 3 * n)
    assert len(C) > 64
    d = rng.standard_normal(len(C))
    K = np.zeros((3 * n + len(C),) * 2)
    for c in range(3):
        K[c * n:(c + 1) * n, c * n:(c + 1) * n] = A
    K[3 * n:, :3 * n], K[:3 * n, 3 * n:] = C, C.T
    ref = np.linalg.solve(K, np.concatenate([b, d]))
    r = T.solveSaddleFromA(A, n, C, b, d)
    assert r["residual"] <= 1e-10
    assert np.linalg.norm(r["x"] - ref[:3 * n]) <= 1e-9 * np.linalg.norm(ref[:3 * n])
    assert np.linalg.norm(r["lambda"] - ref[3 * n:]) <= 1e-9 * max(1.0, np.linalg.norm(ref[3 * n:]))
