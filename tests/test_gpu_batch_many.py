"""Batches of many small problems: the right problem for every item, found in
time that does not grow with the number of problems ahead of it."""
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


def _problem(shape, kernel, seed):
    nz, ny, nx = shape
    n = 14 if kernel == ps.PS_KERNEL_HIMENO19 else 2
    grids = [ps.Grid(shape) for _ in range(n)]
    for i, g in enumerate(grids):
        g.copyin(synth.uniform(shape, seed + i))
    inner = ps.domain(1, nx - 1, 1, ny - 1, 1, nz - 1)
    dom, scalars = {ps.PS_KERNEL_DIFFUSION7: (ps.full_domain(shape), COEF),
                    ps.PS_KERNEL_SUM7: (inner, ()),
                    ps.PS_KERNEL_HIMENO19: (inner, [0.8])}[kernel]
    maps = [ps.stencil_map(kernel, dom, p + grids[2:], scalars)
            for p in (grids[:2], grids[1::-1])]
    return grids, maps


@pytest.mark.parametrize("count", [1, 2, 3, 33, 300])
def test_every_problem_of_many(rt, count):
    rng = np.random.default_rng(count)
    kernels = [ps.PS_KERNEL_DIFFUSION7, ps.PS_KERNEL_SUM7, ps.PS_KERNEL_HIMENO19]
    specs = [(tuple(int(v) for v in rng.integers(3, 24, 3)), kernels[int(rng.integers(3))], 7 * i)
             for i in range(count)]
    batch, alone = [_problem(*s) for s in specs], [_problem(*s) for s in specs]
    b = ps.batch_create([m for _, m in batch])
    ps.batch_run(b, 3)
    for _, m in alone:
        ps.stencil_run(m, 3)
    for (g, _), (h, _) in zip(batch, alone):
        for k in (0, 1):
            assert np.array_equal(g[k].copyout().view(np.uint32), h[k].copyout().view(np.uint32))
    ps.batch_free(b)
    for g, _ in batch + alone:
        for x in g:
            x.free()


def _step(problems):
    """Best time of a step of the batch, in us."""
    b = ps.batch_create([m for _, m in problems])
    ps.batch_run(b, 20)
    times = []
    for _ in range(5):
        ps.lib().PSEventRecord(0)
        ps.batch_run(b, 20)
        ps.lib().PSEventRecord(1)
        times.append(ps.lib().PSEventElapsedMs(0, 1) / 40 * 1e3)
    ps.batch_free(b)
    for g, _ in problems:
        for x in g:
            x.free()
    return min(times)


def test_a_thousand_small_problems(rt):
    # 67 us a step; 190 where a CTA steps over the problems ahead of its item
    # one by one.  A problem of as many cells takes about 20.
    many = _step([_problem((17, 17, 17), ps.PS_KERNEL_SUM7, 0) for _ in range(1000)])
    one = _step([_problem((170, 170, 170), ps.PS_KERNEL_SUM7, 0)])
    assert many < 6 * one
