"""The launches that a context reports (tpe_profile_read) against those that the CUDA profiling
interface sees."""
import ctypes as C

import pytest
import torch

from repulsive_test2_b200 import abi
from repulsive_test2_b200 import api as T
from repulsive_test2_b200 import fixtures as F

pytestmark = pytest.mark.gpu


def _reported():
    ctx = T.context()
    n = (C.c_int64 * (len(abi.KGROUPS) + 1))()
    ms = (C.c_double * (len(abi.KGROUPS) + 1))()
    assert ctx.lib.tpe_profile_read(ctx.ptr, ms, n) == abi.TPE_OK
    return n[len(abi.KGROUPS)]


def _check(call):
    call()
    before = _reported()
    with torch.profiler.profile(activities=[torch.profiler.ProfilerActivity.CUDA]) as p:
        call()
        torch.cuda.synchronize()
    seen = [e for e in p.events() if e.device_type == torch.autograd.DeviceType.CUDA and "Mem" not in e.name]
    assert seen and _reported() - before == len(seen)


# one subtree; one level above the subtrees; the longest sort within a tile, and beyond it
@pytest.mark.parametrize("n", [100, 1500, 4096, 5000, 40000, 131072])
def test_barnes_hut(n):
    v, e = F.trefoil(n)
    _check(lambda: T.bhEnergy(v, e, theta=0.5, leafSize=8))


@pytest.mark.parametrize("n", [128, 2100])
def test_energy_and_gradient(n):
    v, e = F.trefoil(n, jitter=0.01, seed=1)
    _check(lambda: T.calculateEnergy(v, e))
    _check(lambda: T.energyAndGradient(v, e))
