"""Warm-start calls of different sizes from several host threads, each with a
stream and tensors of its own: no call may lower what another one needs."""
import ctypes
import threading

import numpy as np
import pytest

import physis_gb300 as ps

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")
C, TAPS = 16, 27


def _p(t):
    return ctypes.c_void_p(t.data_ptr())


def test_layers_of_different_sizes_side_by_side():
    ps.build()
    ps.init()
    L = ps.lib()
    # shared memory of a CTA: 127, 46, 100 and 68 KB
    sizes = [(2, 3, 31, 31), (1, 2, 3, 3), (2, 2, 25, 25), (3, 4, 9, 9)]
    jobs = []
    for k, dims in enumerate(sizes):
        g = torch.Generator(device="cuda").manual_seed(k)
        n = int(np.prod(dims)) * C
        x = torch.randn(n, generator=g, device="cuda").to(torch.bfloat16)
        w = torch.randn(TAPS * C * C, generator=g, device="cuda").to(torch.bfloat16)
        y = torch.empty_like(x)
        jobs.append((dims, x, w, y, torch.cuda.Stream()))
    torch.cuda.synchronize()
    bad = []

    def call(dims, x, w, y, stream):
        return L.PSWarmStartConv(_p(x), _p(w), None, None, 0, _p(y), None, *dims,
                                 ctypes.c_void_p(stream.cuda_stream))

    alone = []
    for job in jobs:
        assert call(*job) == 0
        torch.cuda.synchronize()
        alone.append(job[3].clone())

    def work(job):
        for _ in range(3000):
            if call(*job):
                bad.append(job[0])
                return

    threads = [threading.Thread(target=work, args=(job,)) for job in jobs]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    torch.cuda.synchronize()
    ps.clear_error()
    assert not bad
    for job, y in zip(jobs, alone):
        assert torch.equal(job[3].view(torch.int16), y.view(torch.int16))
