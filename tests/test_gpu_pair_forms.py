"""The (edge, vertex) pair kernels on the topologies and sizes where they can go
wrong: edges of the 32-vertex masks and 128-thread workers, one and two edges per
thread, runs that break inside a thread, isolated vertices, shared and repeated
edges, hubs (which keep the edge-pair kernels), touching and flat curves, other
exponents and batches.

Against the FP64 oracle at the repository's parity bound, 1e-10 relative: both
sides sum the same terms in FP64, each accurate to a few units in the last
place (times |e||d|/|e x d| <= 1e4 for the flattest triangle of these curves,
2^-53 * 1e4 * 10 = 1e-11), all energy terms positive."""
from __future__ import annotations

import numpy as np
import pytest

import oracle_lib as O
from repulsive_test2_b200 import api as T
from repulsive_test2_b200 import fixtures as F

pytestmark = pytest.mark.gpu
TOL = 1e-10


def _check(v, e, alpha=3.0, beta=6.0):
    e = np.asarray(e, dtype=np.int32)
    en, g = T.energyAndGradient(v, e, alpha, beta)
    ref, gr = O.energy(v, e, alpha, beta), O.gradient(v, e, alpha, beta)
    assert abs(en - ref) <= TOL * abs(ref)
    assert abs(T.calculateEnergy(v, e, None, alpha, beta) - ref) <= TOL * abs(ref)
    assert np.linalg.norm(g - gr) <= TOL * max(np.linalg.norm(gr), 1e-300)
    return g


@pytest.mark.parametrize("n", [3, 4, 5, 31, 33, 127, 128, 129, 260, 1023, 2047, 2048, 2049])
def test_closed_loops(n):
    v, e = F.trefoil(n, jitter=0.01, seed=n)
    if n == 3:  # no disjoint pair
        en, g = T.energyAndGradient(v, e)
        assert en == 0.0 and not g.any()
        return
    _check(v, e)


@pytest.mark.parametrize("alpha,beta", [(2.0, 4.5), (2.7, 5.3)])
@pytest.mark.parametrize("n", [97, 2050])
def test_other_exponents(n, alpha, beta):
    v, e = F.random_walk_knot(n, seed=3)
    _check(v, e, alpha, beta)


def test_runs_broken_anywhere():
    """2100 edges (two per thread) in a shuffled order and with flipped ends, three
    isolated vertices, two repeated edges and one edge from a vertex to itself."""
    v, e = F.loop_network(3, 700, 4, 5)
    rng = np.random.default_rng(1)
    e = e[rng.permutation(len(e))]
    flip = rng.random(len(e)) < 0.5
    e[flip] = e[flip][:, ::-1]
    e = np.concatenate([e, e[:2], [[5, 5]]])
    v = np.concatenate([v[:100], rng.standard_normal((3, 3)), v[100:]])
    e = np.where(e >= 100, e + 3, e)
    g = _check(v, e)
    assert not g[100:103].any()


@pytest.mark.parametrize("spokes", [5, 20, 200])
def test_hub(spokes):
    """A hub of `spokes` chains of four edges: near lists grow with its degree squared
    (200 spokes: the edge-pair kernels)."""
    rng = np.random.default_rng(spokes)
    v, e = [np.zeros(3)], []
    for s in range(spokes):
        d = rng.standard_normal(3)
        d /= np.linalg.norm(d)
        prev = 0
        for k in range(4):
            v.append(d * (k + 1) + 0.05 * rng.standard_normal(3))
            e.append([prev, len(v) - 1])
            prev = len(v) - 1
    _check(np.array(v), e)


def test_touching_and_flat():
    """Two open chains: one straight on integer points (every area of it zero), one
    that passes through one of its vertices and within 1e-11 of another."""
    a = np.stack([np.arange(40.0), np.zeros(40), np.zeros(40)], axis=1)
    b = np.stack([np.full(30, 7.0), np.arange(-15.0, 15.0), np.zeros(30)], axis=1)
    b[20] = [21.0, 1e-11, 0.0]
    v = np.concatenate([a, b])
    e = np.concatenate([np.stack([np.arange(39), np.arange(1, 40)], 1),
                        np.stack([np.arange(40, 69), np.arange(41, 70)], 1)])
    assert (v[40 + 15] == v[7]).all()
    e = e.astype(np.int32)
    en, ref = T.calculateEnergy(v, e), O.energy(v, e)
    assert abs(en - ref) <= 1e-8 * abs(ref)  # 1e-11 from a vertex: the area keeps 1e-16 / 1e-11 of its digits
    en2, _ = T.energyAndGradient(v, e)
    assert abs(en2 - en) <= 1e-8 * abs(ref)


@pytest.mark.parametrize("n,curves", [(50, 1), (301, 7), (2050, 3)])
def test_batches(n, curves):
    v, e = F.random_walk_knot(n, seed=2)
    vs = np.stack([v * (1.0 + 0.1 * c) for c in range(curves)])
    got = T.energyBatch(vs, e)
    for c in range(curves):
        assert abs(got[c] - O.energy(vs[c], e)) <= TOL * got[c]


def test_not_finite():
    v, e = F.trefoil(64, jitter=0.01, seed=1)
    for bad in (np.nan, np.inf):
        w = v.copy()
        w[9, 1] = bad
        assert np.isnan(T.calculateEnergy(w, e)) or np.isinf(T.calculateEnergy(w, e))
