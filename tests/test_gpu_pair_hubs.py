"""Vertices of high degree in the (edge, vertex) pair kernels: near lists longer than the step that
searches them, sums over a hub's edges less those to one of its neighbours (and one by one where
such an edge is most of the sum), hubs next to hubs. Against the oracle at the parity bound of
tests/test_gpu_pair_forms.py; the batch and the repeated call give the same bits."""
import numpy as np
import pytest

import oracle_lib as O
from repulsive_test2_b200 import api as T

pytestmark = pytest.mark.gpu
TOL = 1e-10


def _stars(hubs, spokes, length, seed, far=1.0):
    """A loop (or a line) of hubs, each with `spokes` chains of `length` edges; `far` stretches the
    first edge of each hub's first chain."""
    rng = np.random.default_rng(seed)
    v = [[3 * np.cos(6.28 * i / hubs), 3 * np.sin(6.28 * i / hubs), 0.1 * i] for i in range(hubs)]
    e = [[i, (i + 1) % hubs] for i in range(hubs if hubs > 2 else hubs - 1)]
    for i in range(hubs):
        for s in range(spokes):
            at, d = i, rng.standard_normal(3) * 0.1
            for k in range(length):
                v.append(np.array(v[at]) + d * (far if s == 0 and k == 0 else 1.0) + 0.01 * rng.standard_normal(3))
                e.append([at, len(v) - 1])
                at = len(v) - 1
    e = np.array(e, dtype=np.int32)
    flip = rng.random(len(e)) < 0.3
    e[flip] = e[flip][:, ::-1]
    return np.array(v), e


@pytest.mark.parametrize("alpha,beta", [(3.0, 6.0), (2.0, 4.5)])
@pytest.mark.parametrize("hubs,spokes,length,far", [(1, 8, 12, 1.0), (1, 9, 12, 1.0), (1, 40, 10, 1.0), (1, 40, 10, 1e3),
                                                    (2, 20, 8, 1.0), (2, 20, 8, 1e3), (5, 12, 5, 1.0), (4, 40, 6, 30.0),
                                                    (30, 18, 4, 1.0)])
def test_hubs_against_oracle(hubs, spokes, length, far, alpha, beta):
    v, e = _stars(hubs, spokes, length, 3, far)
    en, g = T.energyAndGradient(v, e, alpha, beta)
    ref, gr = O.energy(v, e, alpha, beta), O.gradient(v, e, alpha, beta)
    one = T.calculateEnergy(v, e, None, alpha, beta)
    assert abs(en - ref) <= TOL * ref and abs(one - ref) <= TOL * ref
    assert np.linalg.norm(g - gr) <= TOL * np.linalg.norm(gr)
    assert np.array_equal(T.energyBatch(np.repeat(v[None], 3, 0), e, alpha, beta), np.full(3, one))
    assert np.array_equal(T.energyAndGradient(v, e, alpha, beta)[1], g)
