"""A call that fails half-way leaves its context fit for the next one: the same bits as a
context that has not failed."""
import numpy as np
import pytest

from repulsive_test2_b200 import abi
from repulsive_test2_b200 import api as T
from repulsive_test2_b200 import fixtures as F

pytestmark = pytest.mark.gpu


def _set(v, e, kind="length"):
    blocks = [T.barycenterBlock(T.barycenterTarget(v, e))]
    return blocks + [T.totalLengthBlock(T.totalLength(v, e)) if kind == "length" else
                     T.edgeLengthsBlock(T.edgeLengths(v, e))]


@pytest.mark.parametrize("kind,precision", [("length", "fp64"), ("length", "mixed"), ("edges", "mixed")])
def test_out_of_memory(kind, precision, monkeypatch):
    """Each growth of a device buffer in a context's first step fails once. The gradient's
    buffers grow before the assembly: its failure may not leave the next call with the edge
    records of the step's positions."""
    v, e = F.trefoil(150, jitter=0.01, seed=1)
    w, _ = F.trefoil(150, jitter=0.01, seed=2)
    dE = F.normals(3, v.size).reshape(-1, 3)
    want = T.solveConstrainedGradientSet(w, e, None, 3.0, 6.0, 1e-10, dE, _set(w, e, kind))
    failed = 0
    for n in range(1, 200):
        ctx = T.Context()
        monkeypatch.setattr(T, "_CTX", ctx)
        assert ctx.lib.tpe_tune(ctx.ptr, abi.TUNE_FAIL_ALLOC, n) == abi.TPE_OK
        try:
            T.sobolevStepSet(v, e, None, _set(v, e, kind), {"projectionMode": "frozen", "precision": precision})
            break  # fewer than n growths
        except T.TpeError:
            failed += 1
        finally:
            ctx.lib.tpe_tune(ctx.ptr, abi.TUNE_FAIL_ALLOC, 0)
        got = T.solveConstrainedGradientSet(w, e, None, 3.0, 6.0, 1e-10, dE, _set(w, e, kind))
        assert np.array_equal(got["gTilde"], want["gTilde"]), n
        ctx.close()
    assert failed > 20


def test_a_topology_that_failed_is_none(monkeypatch):
    """No call runs on the sizes of a topology whose lists are not in place."""
    v, e = F.trefoil(40, jitter=0.01, seed=1)
    w, f = F.trefoil(700, jitter=0.01, seed=2)
    small, large = T.calculateEnergy(v, e), T.calculateEnergy(w, f)
    for n in range(1, 4):  # the topology's three lists
        ctx = T.Context()
        monkeypatch.setattr(T, "_CTX", ctx)
        assert T.calculateEnergy(v, e) == small
        ctx.lib.tpe_tune(ctx.ptr, abi.TUNE_FAIL_ALLOC, n)
        with pytest.raises(T.TpeError):
            T.calculateEnergy(w, f)
        en = np.zeros(1)
        rc = ctx.lib.tpe_energy(ctx.ptr, T._dp(np.zeros((700, 3))), abi.tpe_params(3.0, 6.0, 1e-10), T._dp(en))
        assert rc == abi.TPE_ERR_NO_TOPOLOGY
        assert T.calculateEnergy(v, e) == small
        assert T.calculateEnergy(w, f) == large
        ctx.close()
