"""The Barnes-Hut tree at the size from which the device builds it: subtrees of every size between
its halves, and its longest and shortest leaves."""
import pytest

import test_gpu_bh_tree as B

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,leaf,kind", [(1299, 8, "walk"), (1300, 8, "ladder"), (1300, 1, "walk"), (1300, 512, "walk"),
                                         (2047, 8, "trefoil"), (2048, 1, "ladder"), (2048, 8, "walk")])
def test_either_side(n, leaf, kind):
    B.test_device_tree_is_the_host_tree(n, leaf, kind)
