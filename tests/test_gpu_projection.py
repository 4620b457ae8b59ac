"""The frozen projection of small sets on the device (up to 16 rows) against the loop on the
host, which the search with one trial at a time takes: the same decisions and bits, for every
block kind, at the row limit and beyond it, with the iteration cap at 0, 1 and not a multiple of
the look-ahead."""
import numpy as np
import pytest

from repulsive_test2_b200 import api as T
from repulsive_test2_b200 import fixtures as F

pytestmark = pytest.mark.gpu


def _blocks(v, e, kind):
    points = [T.pointBlock(i * len(v) // 8, v[i * len(v) // 8] + 1e-3) for i in range(5)]
    length = T.totalLengthBlock(T.totalLength(v, e))
    center = T.barycenterBlock(T.barycenterTarget(v, e))
    return {"length": [length], "center": [center], "both": [center, length], "point": points[:1],
            "rows16": [center, length] + points[:4], "rows19": [center, length] + points}[kind]


@pytest.mark.parametrize("kind", ["length", "center", "both", "point", "rows16", "rows19"])
@pytest.mark.parametrize("V,cap,trials", [(24, 8, 3), (301, 0, 4), (301, 1, 16), (512, 7, 8), (512, 8, 16)])
def test_device_projection_is_the_host_projection(kind, V, cap, trials):
    v, e = F.random_walk_knot(V, seed=2)
    o = {"projectionMode": "frozen", "projection": {"maxIter": cap}}
    seq = T.sobolevStepSet(v, e, None, _blocks(v, e, kind), {**o, "trials": 1})
    bat = T.sobolevStepSet(v, e, None, _blocks(v, e, kind), {**o, "trials": trials})
    for key in ("tau", "projectionIterations", "reason"):
        assert bat["stats"].get(key) == seq["stats"].get(key)
    assert bat["accepted"] == seq["accepted"] and bat["energy"] == seq["energy"]
    assert np.array_equal(bat["vertices"], seq["vertices"])
