"""The mixed mode with the FP64 factor (up to 5000 vertices) and, beyond that, with the
FP32 factor: both against the FP64 step, at a residual that one solve reaches and at one that
needs a correction. Tolerances: those of the mixed mode (gradient 1e-6, energy 1e-8)."""
import numpy as np
import pytest

from repulsive_test2_b200 import api as T
from repulsive_test2_b200 import fixtures as F

pytestmark = pytest.mark.gpu


def _step(v, e, **opts):
    blocks = [T.barycenterBlock(T.barycenterTarget(v, e)), T.totalLengthBlock(T.totalLength(v, e))]
    return T.sobolevStepSet(v, e, None, blocks, {"projectionMode": "frozen", "collectField": True, **opts})


@pytest.mark.parametrize("V,tol,its", [(24, 1e-9, {1}), (63, 1e-17, {2, 3}), (64, 1e-17, {2, 3}), (777, 1e-9, {1}),
                                       (2801, 1e-9, {1}), (5000, 1e-17, {2, 3}), (5001, 1e-12, set(range(1, 61)))])
def test_mixed_with_either_factor(V, tol, its):
    # (a jitter of 0.01 exceeds the spacing of 5000 vertices: FP32 factors break down on some)
    v, e = F.trefoil(V, jitter=0.01, seed=V) if V <= 5000 else F.random_walk_knot(V, seed=1)
    r64 = _step(v, e, precision="fp64")
    r = _step(v, e, precision="mixed", refineTol=tol)
    assert r["stats"]["refineIterations"] in its
    assert r["stats"]["tau"] == r64["stats"]["tau"] and r["accepted"] == r64["accepted"]
    g64, g = r64["descentField"], r["descentField"]
    assert np.linalg.norm(g - g64) <= 1e-6 * np.linalg.norm(g64)
    assert abs(r["energy"] - r64["energy"]) <= 1e-8 * abs(r64["energy"])


def test_a_residual_out_of_reach_is_the_fp64_step():
    v, e = F.trefoil(200, jitter=0.01, seed=3)
    r64 = _step(v, e, precision="fp64")
    r = _step(v, e, precision="mixed", refineTol=1e-300, refineMaxIter=2)
    assert r["stats"]["refineIterations"] == -1
    assert np.array_equal(r["vertices"], r64["vertices"])
