"""Which diffusion runs take the one launch: where an estimate of its time, blocks
of rows cut short and passes over more blocks than threads counted, beats that of
sweeps."""
import numpy as np
import pytest

import physis_gb300 as ps
from physis_gb300 import synth

pytestmark = pytest.mark.gpu
COEF = (0.1,) * 6 + (0.4,)


@pytest.fixture(scope="module")
def rt():
    ps.build()
    ps.init()
    yield ps
    ps.clear_error()


@pytest.mark.parametrize("shape,dtype,one", [
    # one launch 22 us a step, sweeps 15; 6.4 and 5.7
    ((9, 110, 278), np.float64, False), ((124, 124, 124), np.float32, False),
    ((64, 64, 64), np.float32, True), ((120, 120, 120), np.float32, True),
    ((48, 48, 48), np.float64, True), ((72, 72, 72), np.float64, True)])
def test_one_launch_or_sweeps(rt, shape, dtype, one):
    a = synth.uniform(shape, 1).astype(dtype)
    grids = [ps.Grid(shape, dtype) for _ in range(2)]
    for g in grids:
        g.copyin(a)
    run = [ps.stencil_map(ps.PS_KERNEL_DIFFUSION7, ps.full_domain(shape), p, COEF)
           for p in (grids, grids[::-1])]
    before = ps.launch_count()
    ps.stencil_run(run, 50)
    launches = ps.launch_count() - before
    for g in grids:
        g.free()
    assert (launches == 1) == one
