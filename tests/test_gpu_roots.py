"""The roots that the FP64 pair kernels form from a hardware or FP32 estimate and a series, over
the whole range that they are taken for: against extended precision, with the bound that their
roundings give (units of 2^-53, relative), and against CUDA's own function."""
import numpy as np
import pytest
import torch

from repulsive_test2_b200 import abi
from repulsive_test2_b200 import api as T

pytestmark = pytest.mark.gpu
U = 2.0 ** -53


def _roots(which, x):
    ctx = T.context()
    d = torch.tensor(x, dtype=torch.float64, device="cuda")
    out = torch.zeros(len(x), 2, dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    assert ctx.lib.tpe_root_check(ctx.ptr, which, d.data_ptr(), len(x), out.data_ptr()) == abi.TPE_OK
    return out.cpu().numpy().T


def _samples(lo, hi, n=1 << 20):
    """Log-uniform between the powers of ten, with powers of two and their neighbours."""
    rng = np.random.default_rng(7)
    x = 10.0 ** rng.uniform(lo, hi, n)
    p = 2.0 ** np.arange(np.ceil(lo / np.log10(2.0)), np.floor(hi / np.log10(2.0)))
    return np.concatenate([x, p, np.nextafter(p, np.inf), np.nextafter(p, 0.0)[1:]])


def _err(got, exact):
    return float(np.max(np.abs((np.longdouble(got) - exact) / exact)))


# x^(-1/3): the last sum rounds (1) and the product x y, of which a third counts; CUDA's rcbrt is
# within one unit in the last place (2). Narrow ranges at the ends, where the estimate is worst.
@pytest.mark.parametrize("lo,hi", [(-30, 30), (-30, -29.5), (29.5, 30), (-17, -13), (-1, 1), (-60, -30), (30, 200)])
def test_inverse_cube_root(lo, hi):
    x = _samples(lo, hi)
    own, cuda = _roots(abi.ROOT_INV_CBRT, x)
    exact = 1.0 / np.cbrt(np.longdouble(x))
    assert _err(own, exact) <= (1.34 if -30 <= lo and hi <= 30 else 2.0) * U
    assert _err(cuda, exact) <= 2.0 * U


# x^(-1/2): the last sum rounds (1), the product x y rounds and half of it counts, the e^3 left out is
# 5/16 2^-57 (0.02). 1/x: the last sum, and e^3 of 2^-57 (0.07). Every normal number whose result is one.
@pytest.mark.parametrize("which,bound", [(abi.ROOT_RSQRT, 1.53), (abi.ROOT_RECIP, 1.08)])
@pytest.mark.parametrize("lo,hi", [(-307.6, 307.6), (-307.6, -300), (300, 307.6), (-1, 1)])
def test_hardware_estimates(which, bound, lo, hi):
    x = _samples(lo, hi)
    own, cuda = _roots(which, x)
    exact = 1.0 / (np.sqrt(np.longdouble(x)) if which == abi.ROOT_RSQRT else np.longdouble(x))
    assert _err(own, exact) <= bound * U
    assert _err(cuda, exact) <= (2.0 if which == abi.ROOT_RSQRT else 1.0) * U


def test_beyond_normal_numbers():
    """What rsqrt_normal's callers rely on: no finite result there."""
    own, _ = _roots(abi.ROOT_RSQRT, np.array([0.0, 5e-324, 2e-308, np.inf, np.nan, -1.0]))
    assert not np.isfinite(own).any()
