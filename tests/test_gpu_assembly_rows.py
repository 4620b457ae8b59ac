"""The closed-loop Gram assembly at the sizes where its rows per warp change (4, 8, 16, 32, 64),
against the general assembly: 1e-12 of the matrix norm, as tests/test_gpu_assembly_forms.py."""
import numpy as np
import pytest

from repulsive_test2_b200 import api as T
from repulsive_test2_b200 import fixtures as F

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [549, 550, 1199, 1200, 1217, 1899, 1900, 1951, 7001])
def test_loop_against_general(n):
    v, e = F.random_walk_knot(n, seed=n) if n % 2 else F.trefoil(n, jitter=0.01, seed=n)
    A = np.asarray(T.assembleAFlat(v, e)).reshape(n, n)
    G = np.asarray(T.assembleBHighFlat(v, e)).reshape(n, n)
    G += np.asarray(T.assembleBLowFlat(v, e)).reshape(n, n)
    assert np.array_equal(A, A.T)
    assert np.linalg.norm(A - G) <= 1e-12 * np.linalg.norm(G)
