"""Energy and gradient over the scales at which their terms are in the double range. With eps = 0
the exponents (2, 4) leave an energy as it is when its curve grows by s and its gradient falls by
s; (3, 6) divides them by s and s^2. s a power of two, so that all but the general powers scale
exactly: those are within two units in the last place, and the sums hold some 1e3 times that."""
import numpy as np
import pytest

from repulsive_test2_b200 import api as T
from repulsive_test2_b200 import fixtures as F

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [33, 700, 2050])
@pytest.mark.parametrize("alpha,beta,power", [(2.0, 4.0, 100), (2.0, 4.0, 200), (2.0, 4.0, 240), (2.0, 4.0, 250),
                                              (2.0, 4.0, 252), (3.0, 6.0, 100), (3.0, 6.0, 130), (3.0, 6.0, 155), (3.0, 6.0, 162)])
def test_large_curves(n, alpha, beta, power):
    v, e = F.trefoil(n, jitter=0.01, seed=2)
    s = 2.0 ** power
    down = 1.0 if alpha == 2.0 else s
    e0, g0 = T.energyAndGradient(v, e, alpha, beta, 0.0)
    e1, g1 = T.energyAndGradient(v * s, e, alpha, beta, 0.0)
    assert abs(e1 * down - e0) <= 1e-12 * e0
    assert np.linalg.norm(g1 * down * s - g0) <= 1e-12 * np.linalg.norm(g0)
