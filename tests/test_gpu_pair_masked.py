"""Pairs of edges that share a vertex are left out whatever their values: coincident neighbours
without an epsilon (a distance of zero to a negative power), and vertices that are no numbers on
edges that no other edge is disjoint from. Against the oracle, at the parity bound of
tests/test_gpu_pair_forms.py."""
import numpy as np
import pytest

import oracle_lib as O
from repulsive_test2_b200 import api as T
from repulsive_test2_b200 import fixtures as F

pytestmark = pytest.mark.gpu
TOL = 1e-10


@pytest.mark.parametrize("alpha,beta", [(3.0, 6.0), (2.0, 4.5)])
@pytest.mark.parametrize("n", [6, 34, 140, 700, 2100])
def test_coincident_leaves(n, alpha, beta):
    """An open curve with two ends at one place on its last vertex."""
    v, _ = F.trefoil(n, jitter=0.01, seed=3)
    v[n - 1] = v[n - 2]
    e = np.array([[i, i + 1] for i in range(n - 2)] + [[n - 3, n - 1]], dtype=np.int32)
    en, g = T.energyAndGradient(v, e, alpha, beta, 0.0)
    ref, gr = O.energy(v, e, alpha, beta, 0.0), O.gradient(v, e, alpha, beta, 0.0)
    assert abs(en - ref) <= TOL * ref and abs(T.calculateEnergy(v, e, None, alpha, beta, 0.0) - ref) <= TOL * ref
    assert np.linalg.norm(g - gr) <= TOL * np.linalg.norm(gr)


@pytest.mark.parametrize("bad", [np.nan, np.inf])
@pytest.mark.parametrize("spokes", [1, 2, 20])
def test_no_disjoint_pair(spokes, bad):
    rng = np.random.default_rng(spokes)
    v = rng.standard_normal((spokes + 1, 3))
    v[1, 0] = bad
    e = np.array([[0, i + 1] for i in range(spokes)] + [[1, 0]], dtype=np.int32)  # (one edge twice, turned)
    assert T.calculateEnergy(v, e) == 0.0
    en, g = T.energyAndGradient(v, e)
    assert en == 0.0 and not g.any()


def test_a_pair_that_counts_still_shows():
    v, e = F.trefoil(64, jitter=0.01, seed=3)
    v[9, 1] = np.nan
    assert np.isnan(T.calculateEnergy(v, e))
    en, g = T.energyAndGradient(v, e)
    assert np.isnan(en) and np.isnan(g).any()
