"""The convolution's two forms on either side of the rule between them: few
slabs of wide planes go to the gathering one, more of them (and the largest
padded planes) to the padded-slab one."""
import pytest

import test_gpu_warmstart_edges as base

pytestmark = pytest.mark.gpu
rt = base.rt


@pytest.mark.parametrize("dims", [(153, 1, 31, 31), (153, 1, 3, 255), (2, 10, 4, 200),
                                  (4, 20, 4, 200), (1, 8, 25, 25), (60, 1, 25, 25), (1, 2, 23, 26)])
@pytest.mark.parametrize("masked", [False, True])
def test_conv_on_both_sides_of_the_rule(rt, dims, masked):
    base.test_conv_edges(rt, dims, masked)
