"""The Barnes-Hut tree as the device builds it: the energy's counts over the host builder's tree
(tpe_edge_tree, which is checked node by node against the reference), traversed here, have to be
the device's exactly and the energy to 1e-12, at the edges of the builder's blocks (subtrees of
1024 edges, sorted tiles of 2048) and with many equal sort keys."""
import ctypes as C

import numpy as np
import pytest

from repulsive_test2_b200 import abi
from repulsive_test2_b200 import api as T
from repulsive_test2_b200 import fixtures as F

pytestmark = pytest.mark.gpu
EPS = 1e-10


def _host_tree(v, e, leaf):
    E = len(e)
    f, i = np.zeros((4 * E + 8, 9)), np.zeros((4 * E + 8, 4), dtype=np.int32)
    perm, nn = np.zeros(E, dtype=np.int32), C.c_int32(0)
    rc = abi.load_library().tpe_edge_tree(
        v.ctypes.data_as(abi.dp), len(v), e.ctypes.data_as(abi.ip), E, EPS, leaf, len(f),
        f.ctypes.data_as(abi.dp), i.ctypes.data_as(abi.ip), perm.ctypes.data_as(abi.ip), C.byref(nn))
    assert rc == 0
    return f, i, perm


def _traverse(v, e, leaf, alpha, beta, theta, theta_t):
    f, ni, perm = _host_tree(v, e, leaf)
    E = len(e)
    a, b = v[e[:, 0]], v[e[:, 1]]
    d, mid = b - a, 0.5 * (a + b)
    ell = np.sqrt((d ** 2).sum(1)) + EPS
    where = np.empty(E, dtype=np.int64)
    where[perm] = np.arange(E)

    def term(I, p, q):  # edges I, their endpoints p, against points q (same length)
        x = p - q
        cn = np.sqrt((np.cross(d[I], x) ** 2).sum(-1)) + EPS
        return cn ** alpha / (np.sqrt((x ** 2).sum(-1)) + EPS) ** beta

    visits = approx = direct = 0
    total = 0.0
    deg = [[] for _ in range(len(v))]
    for J, (p, q) in enumerate(e):
        deg[p].append(where[J])
        deg[q].append(where[J])
    wide = max(len(x) for x in deg)
    inc = np.full((len(v), wide), -1)
    for k, x in enumerate(deg):
        inc[k, :len(x)] = x
    stack = [(0, np.arange(E))]
    while stack:
        n, I = stack.pop()
        begin, count, left, right = ni[n]
        visits += len(I)
        dist = np.sqrt(((mid[I] - f[n, :3]) ** 2).sum(1))
        with np.errstate(divide="ignore", invalid="ignore"):
            ok = (count >= 2) & (dist > 0) & (f[n, 7] / dist <= theta) & (f[n, 8] <= theta_t)
        at = np.concatenate([inc[e[I, 0]], inc[e[I, 1]]], axis=1)
        ok &= ~((at >= begin) & (at < begin + count)).any(1)
        A = I[ok]
        approx += count * len(A)
        c = np.broadcast_to(f[n, :3], (len(A), 3))
        total += (0.5 * ell[A] ** (1 - alpha) * f[n, 6] * (term(A, a[A], c) + term(A, b[A], c))).sum()
        I = I[~ok]
        if len(I) == 0:
            continue
        if left >= 0:
            stack += [(left, I), (right, I)]
            continue
        for J in perm[begin:begin + count]:
            K = I[~((e[I] == e[J, 0]) | (e[I] == e[J, 1])).any(1)]
            direct += len(K)
            s = sum(term(K, p[K], np.broadcast_to(q[J], (len(K), 3))) for p in (a, b) for q in (a, b))
            total += (0.25 * ell[K] ** (1 - alpha) * ell[J] * s).sum()
    return 0.5 * total, [visits, approx, direct]


def _ladder(n):
    """A closed zigzag on a lattice: coordinates and tangents repeat, one of them as -0."""
    k = np.arange(n)
    v = np.stack([np.minimum(k, n - k) // 2 * 0.5, (k % 4 // 2) * 1.0, np.where(k % 3, 0.0, -0.0)], axis=1)
    v[n // 2:, 2] += 2.0
    return np.ascontiguousarray(v), F.closed_edges(n)


@pytest.mark.parametrize("n,leaf,kind", [(3, 1, "walk"), (9, 8, "walk"), (1000, 1, "ladder"), (1024, 8, "walk"),
                                         (1025, 8, "ladder"), (2049, 512, "walk"), (2049, 513, "walk"),
                                         (4100, 8, "ladder"), (5001, 3, "trefoil")])
def test_device_tree_is_the_host_tree(n, leaf, kind):
    v, e = {"walk": lambda: F.random_walk_knot(n, seed=3), "ladder": lambda: _ladder(n),
            "trefoil": lambda: F.trefoil(n, jitter=0.001, seed=3)}[kind]()
    v, e = np.ascontiguousarray(v, dtype=np.float64), np.ascontiguousarray(e, dtype=np.int32)
    for alpha, beta in ((3.0, 6.0), (2.0, 4.5)):
        want, counts = _traverse(v, e, leaf, alpha, beta, 0.5, 0.75)
        got, st = T.bhEnergy(v, e, alpha, beta, EPS, theta=0.5, leafSize=leaf, thetaT=0.75)
        assert [st["visits"], st["approximated_edge_refs"], st["direct_pairs"]] == counts
        assert abs(got - want) <= 1e-12 * abs(want)
