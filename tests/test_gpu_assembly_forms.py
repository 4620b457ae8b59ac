"""The closed-loop Gram assembly (one warp per strip of 30 columns and block of 4 to 64
rows) at the edges of its strips, blocks, batches of 16 rows and size rules, against the
general assembly of the same curve (B + B0 from the edge-pair matrix), and both against
the oracle at small sizes.

Tolerance 1e-12 of the matrix norm, the repository's bound for A: both sides sum the
same terms, each to a few units in the last place."""
from __future__ import annotations

import numpy as np
import pytest

import oracle_lib as O
from repulsive_test2_b200 import api as T
from repulsive_test2_b200 import fixtures as F

pytestmark = pytest.mark.gpu
SIZES = [8, 9, 15, 16, 17, 29, 30, 31, 32, 33, 60, 61, 64, 65, 399, 400, 401, 1399, 1400, 1439, 3071, 3072, 3105]


@pytest.mark.parametrize("n", SIZES)
def test_loop_against_general(n):
    v, e = F.random_walk_knot(n, seed=n) if n % 2 else F.trefoil(n, jitter=0.01, seed=n)
    A = T.assembleAFlat(v, e)
    G = T.assembleBHighFlat(v, e) + T.assembleBLowFlat(v, e)
    assert np.array_equal(A, A.T)
    assert np.linalg.norm(A - G) <= 1e-12 * np.linalg.norm(G)
    if n <= 65:
        R = O.assemble(v, e)
        assert np.linalg.norm(A - R) <= 1e-12 * np.linalg.norm(R)


@pytest.mark.parametrize("n,alpha,beta", [(33, 2.0, 4.5), (401, 2.7, 5.3)])
def test_loop_other_exponents(n, alpha, beta):
    v, e = F.trefoil(n, jitter=0.01, seed=n)
    A = T.assembleAFlat(v, e, None, alpha, beta)
    G = T.assembleBHighFlat(v, e, None, alpha, beta) + T.assembleBLowFlat(v, e, None, alpha, beta)
    assert np.linalg.norm(A - G) <= 1e-12 * np.linalg.norm(G)


def test_loop_touching_vertices():
    """Two vertices far apart along the curve in one place, and one 1e-11 from another."""
    v, e = F.trefoil(64, jitter=0.01, seed=5)
    v[40] = v[7]
    v[50] = v[20] + np.array([1e-11, 0.0, 0.0])
    A, R = T.assembleAFlat(v, e), O.assemble(v, e)
    assert np.linalg.norm(A - R) <= 1e-9 * np.linalg.norm(R)  # 1e-11 + eps keeps 1e-16 / 1e-10 of its digits
