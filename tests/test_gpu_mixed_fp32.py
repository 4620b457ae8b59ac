"""The mixed mode with its FP32 factor at the sizes that take the FP64 one by default: the tests of
the mixed mode once more with the threshold at zero. Each has to have launched the FP32 diagonal
blocks (as the CUDA profiling interface sees it)."""
import pytest
import torch

from repulsive_test2_b200 import abi
from repulsive_test2_b200 import api as T
from test_gpu_mixed import (  # noqa: F401
    test_mixed_against_oracle_small,
    test_mixed_matches_fp64_step,
    test_mixed_non_power_of_two_size,
    test_mixed_refine_cap_falls_back_to_fp64,
    test_repeated_steps_are_bit_identical,
)
from test_gpu_trajectory import test_mixed_steps_against_oracle, traj  # noqa: F401

pytestmark = pytest.mark.gpu


@pytest.fixture(autouse=True)
def fp32_factor(request):
    ctx = T.context()
    assert ctx.lib.tpe_tune(ctx.ptr, abi.TUNE_MIXED_DIRECT, 0) == abi.TPE_OK
    try:
        with torch.profiler.profile(activities=[torch.profiler.ProfilerActivity.CUDA]) as p:
            yield
            torch.cuda.synchronize()
    finally:
        ctx.lib.tpe_tune(ctx.ptr, abi.TUNE_MIXED_DIRECT, -1)
    if "fp64" not in request.node.name.split("[")[-1]:
        assert any("potrf128_kernel" in e.name for e in p.events())
