"""The bounded waits of the FP64 factorization and its triangular solves: one thread block alone
finishes (it does the other blocks' tiles itself, and only polls with nothing to do count against
the limit), and a wait that runs out is an error after which the context gives the same bits."""
import numpy as np
import pytest

from repulsive_test2_b200 import abi
from repulsive_test2_b200 import api as T
from repulsive_test2_b200 import fixtures as F

pytestmark = pytest.mark.gpu


@pytest.fixture
def ctx(monkeypatch):
    c = T.Context()
    monkeypatch.setattr(T, "_CTX", c)
    yield c
    c.close()


def _tune(ctx, **kw):
    names = {"blocks": abi.TUNE_FACTOR_BLOCKS, "polls": abi.TUNE_FACTOR_POLLS, "solve": abi.TUNE_SOLVE_POLLS}
    for k, value in kw.items():
        assert ctx.lib.tpe_tune(ctx.ptr, names[k], value) == abi.TPE_OK


def _call(n, kind, precision="fp64"):
    """length: factor, forward solves and back substitution; edges: inverses (mixed: their blocks)."""
    v, e = F.trefoil(n, jitter=0.01, seed=1)
    blocks = [T.barycenterBlock(T.barycenterTarget(v, e))]
    blocks.append(T.totalLengthBlock(T.totalLength(v, e)) if kind == "length" else
                  T.edgeLengthsBlock(T.edgeLengths(v, e)))
    if precision == "fp64":
        dE = F.normals(3, v.size).reshape(-1, 3)
        return lambda: T.solveConstrainedGradientSet(v, e, None, 3.0, 6.0, 1e-10, dE, blocks)["gTilde"]
    opts = {"projectionMode": "frozen", "precision": precision}
    return lambda: T.sobolevStepSet(v, e, None, blocks, opts)["vertices"]


@pytest.mark.parametrize("n,kind", [(40, "length"), (65, "length"), (129, "length"), (777, "length"), (1500, "length"),
                                    (70, "edges"), (300, "edges"), (650, "edges")])
def test_one_block_finishes(ctx, n, kind):
    """Waits of at most four times the polls after which the block begins to help: at 777 rows it takes
    ten and more tiles in one of them."""
    call = _call(n, kind)
    want = call()
    for blocks in (1, 2, 7):
        _tune(ctx, blocks=blocks, polls=4 * 8192)
        assert np.array_equal(call(), want), blocks


@pytest.mark.parametrize("n,kind,precision", [(777, "length", "fp64"), (300, "length", "mixed"), (300, "edges", "fp64"),
                                              (300, "edges", "mixed")])
def test_factorization_timeout(ctx, n, kind, precision):
    call = _call(n, kind, precision)
    want = call()
    _tune(ctx, polls=1)
    with pytest.raises(T.TpeError, match="factorization kernel ran out"):
        call()
    _tune(ctx, polls=0)
    assert np.array_equal(call(), want)


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_solve_timeout(ctx, precision):
    call = _call(777, "length", precision)
    want = call()
    _tune(ctx, solve=1)
    with pytest.raises(T.TpeError, match="triangular solve ran out"):
        call()
    _tune(ctx, solve=0)
    assert np.array_equal(call(), want)
