"""A mixed step whose FP64 factor breaks down: the FP32 factor has its turn, and where that breaks
down too the step is the FP64 step, singular with its start's vertices."""
import numpy as np
import pytest
import torch

from repulsive_test2_b200 import api as T
from repulsive_test2_b200 import fixtures as F

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [128, 300])
def test_both_factors_break_down(n):
    v, e = F.trefoil(n, jitter=0.01, seed=1)
    v = v.copy()
    v[n // 2:] *= 1e6  # weights fall with distance: pivots of half the curve vanish beside the others'
    blocks = [T.barycenterBlock(T.barycenterTarget(v, e)), T.totalLengthBlock(T.totalLength(v, e))]
    with torch.profiler.profile(activities=[torch.profiler.ProfilerActivity.CUDA]) as p:
        r = T.sobolevStepSet(v, e, None, blocks, {"projectionMode": "frozen", "precision": "mixed"})
        torch.cuda.synchronize()
    names = [x.name for x in p.events()]
    assert any("chol_dag_kernel" in x for x in names) and any("potrf128_kernel" in x for x in names)
    r64 = T.sobolevStepSet(v, e, None, blocks, {"projectionMode": "frozen", "precision": "fp64"})
    for s in (r, r64):
        assert not s["accepted"] and "singular_system" in (s.get("reason"), s["stats"].get("reason"))
        assert np.array_equal(s["vertices"], v)
    assert r["stats"]["refineIterations"] == -1
    # the context is fit for the next step
    w, f = F.trefoil(n, jitter=0.01, seed=2)
    blocks = [T.barycenterBlock(T.barycenterTarget(w, f)), T.totalLengthBlock(T.totalLength(w, f))]
    assert T.sobolevStepSet(w, f, None, blocks, {"projectionMode": "frozen", "precision": "mixed"})["accepted"]
