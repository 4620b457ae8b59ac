"""An energy is the same to the last bit whether its curve is alone in a launch or one of many:
differences of energies from launches of different sizes (finite differences, a caller's own
search over a batch) then hold no other rounding than that of the curves themselves. One and two
edges per thread, chunks of 8 to 128 vertices, groups of one chunk and of many."""
import numpy as np
import pytest

from repulsive_test2_b200 import api as T
from repulsive_test2_b200 import fixtures as F

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [33, 128, 777, 1311, 2050, 5001])
@pytest.mark.parametrize("alpha,beta", [(3.0, 6.0), (2.0, 4.5)])
def test_batch_is_the_single_curve(n, alpha, beta):
    v, e = F.random_walk_knot(n, seed=3)
    one = T.calculateEnergy(v, e, None, alpha, beta)
    for count in (1, 2, 16, 37, 130) + ((512,) if n < 1000 else ()):
        got = T.energyBatch(np.repeat(v[None], count, 0), e, alpha, beta)
        assert np.array_equal(got, np.full(count, one)), count


def test_batch_of_a_network():
    v, e = F.loop_network(loops=3, n=400, junctions=4, seed=5)
    one = T.calculateEnergy(v, e)
    assert np.array_equal(T.energyBatch(np.repeat(v[None], 40, 0), e), np.full(40, one))


@pytest.mark.parametrize("n", [128, 777])
def test_finite_differences_are_those_of_the_single_energies(n):
    """Components from the first, a middle and the last (shorter) launch."""
    v, e = F.random_walk_knot(n, seed=4)
    g = T.gradientFiniteDiff(v, e).ravel()
    e0 = T.calculateEnergy(v, e)
    for i in (0, 200, 3 * n // 2, 3 * n - 1):
        w = v.ravel().copy()
        w[i] += 1e-6
        assert g[i] == (T.calculateEnergy(w.reshape(-1, 3), e) - e0) / 1e-6
