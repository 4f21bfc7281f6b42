"""Point stencils whose ring needs tiles of one or two rows, with halos wider
than what a producer fetches ahead: offsets of up to 4 in every direction."""
import numpy as np
import pytest

import test_gpu_points as base

pytestmark = pytest.mark.gpu
rt, kernel_form = base.rt, base.kernel_form

# (seed, shape, dtype, boundary, points, radius, weighted, shrink)
WIDE = [(61, (13, 21, 70), np.float32, 1, 25, 4, True, False),
        (62, (12, 40, 131), np.float32, 2, 64, 4, True, True),
        (63, (17, 19, 66), np.float64, 1, 33, 4, True, False),
        (64, (11, 70, 35), np.int64, 2, 64, 4, False, False),
        (65, (9, 5, 9), np.float32, 1, 64, 4, True, False),
        (66, (30, 33, 40), np.float32, 0, 64, 2, True, False),
        (67, (10, 65, 129), np.float64, 2, 48, 2, True, False),
        (68, (10, 65, 129), np.int32, 1, 64, 2, False, True),
        (69, (1, 90, 300), np.float64, 1, 25, 2, True, False),
        (70, (40, 9, 33), np.float32, 2, 40, 4, False, False)]


@pytest.mark.parametrize("seed,shape,dtype,boundary,npts,radius,weighted,shrink", WIDE)
def test_wide_point_stencils_bit_exact(rt, oracle, kernel_form, seed, shape, dtype, boundary, npts,
                                       radius, weighted, shrink):
    base.test_random_point_stencils_bit_exact(rt, oracle, kernel_form, seed, shape, dtype, boundary,
                                              npts, radius, weighted, shrink)
