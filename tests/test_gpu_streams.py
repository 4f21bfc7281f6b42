"""The order between the runtime's stream and CUDA's default one, which is
PyTorch's and the PSWarmStart* calls': whichever is busy, work issued later on
the other sees what was issued before."""
import ctypes

import numpy as np
import pytest

import physis_gb300 as ps

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

COEF = (0.1,) * 6 + (0.4,)
BUSY = 20_000_000  # cycles, about 10 ms
TAPS, C = 27, 16


@pytest.fixture(scope="module")
def rt():
    ps.build()
    ps.init()
    yield ps
    ps.clear_error()


@pytest.fixture(scope="module")
def sweeps(rt):
    # a call that keeps the runtime's stream busy for milliseconds
    grids = [ps.Grid((256, 512, 512)) for _ in range(2)]
    for g in grids:
        g.copyin(np.ones(g.shape, np.float32))
    dom = ps.full_domain(grids[0].shape)
    maps = [ps.stencil_map(ps.PS_KERNEL_DIFFUSION7, dom, p, COEF) for p in (grids, grids[::-1])]
    yield lambda: ps.stencil_run(maps, 50)
    for g in grids:
        g.free()


def _p(t):
    return ctypes.c_void_p(t.data_ptr())


def _handle(explicit):
    return ctypes.c_void_p(1) if explicit else None  # 1: cudaStreamLegacy


def _weights(seed):
    w = torch.randn((TAPS, C, C), generator=torch.Generator().manual_seed(seed))
    return w, w.to(torch.bfloat16).transpose(1, 2).contiguous()


@pytest.mark.parametrize("explicit", [False, True])
def test_torch_reads_what_a_call_behind_sweeps_wrote(rt, sweeps, explicit):
    w, fwd = _weights(1)
    dw, wf, wb = w.cuda(), torch.zeros_like(fwd, device="cuda"), torch.zeros_like(fwd, device="cuda")
    torch.cuda.synchronize()
    sweeps()
    assert ps.lib().PSWarmStartPrepareWeights(_p(dw), _p(wf), _p(wb), _handle(explicit)) == 0
    assert torch.equal(wf.cpu(), fwd)


@pytest.mark.parametrize("explicit", [False, True])
def test_a_call_reads_what_torch_wrote_late(rt, explicit):
    w, fwd = _weights(2)
    src, dw = w.cuda(), torch.zeros_like(w, device="cuda")
    wf, wb = torch.zeros_like(fwd, device="cuda"), torch.zeros_like(fwd, device="cuda")
    torch.cuda.synchronize()
    torch.cuda._sleep(BUSY)
    dw.copy_(src)
    assert ps.lib().PSWarmStartPrepareWeights(_p(dw), _p(wf), _p(wb), _handle(explicit)) == 0
    ps.synchronize()
    assert torch.equal(wf.cpu(), fwd)


def test_a_repeated_weight_gradient_is_waited_for(rt, sweeps):
    dims = (3, 5, 9, 9)
    n = int(np.prod(dims)) * C
    gen = torch.Generator(device="cuda").manual_seed(3)
    x = torch.randn(n, generator=gen, device="cuda").to(torch.bfloat16)
    dy = torch.randn(n, generator=gen, device="cuda").to(torch.bfloat16)
    work = torch.empty(4 * (TAPS * C * C + C), device="cuda")
    got = []
    for _ in range(2):
        dw = torch.full((TAPS, C, C), float("nan"), device="cuda")
        db = torch.full((C,), float("nan"), device="cuda")
        torch.cuda.synchronize()
        sweeps()
        assert ps.lib().PSWarmStartWeightGrad(_p(x), _p(dy), _p(work), 4, _p(dw), _p(db), *dims,
                                              None) == 0
        got.append((dw.cpu(), db.cpu()))
    assert all(torch.isfinite(t).all() for t in got[0])
    assert torch.equal(got[0][0], got[1][0]) and torch.equal(got[0][1], got[1][1])


def test_sweeps_then_pool_then_network(rt, sweeps):
    # the runtime's sweeps, a NULL-stream call and PyTorch's stream in turn,
    # without a synchronisation, as one program issues them
    from physis_gb300 import warmstart as ws
    shape = (33, 17, 17)
    st = ws.Stack([ws.make_instance(np.random.default_rng(4), shape)], shape, nsx=1)
    zc, yc, xc = ws.coarse_shape(shape, 4)
    net, f = ws.Net(5), st.fields(4)
    got = []
    for busy in (False, True):
        x = torch.zeros(zc * yc * xc * C, dtype=torch.bfloat16, device="cuda")
        torch.cuda.synchronize()
        if busy:
            sweeps()
        assert ps.lib().PSWarmStartPool(ctypes.byref(f), _p(x), None) == 0
        if not busy:
            ps.synchronize()
        got.append(net.forward(x, (1, zc, yc, xc)).cpu())
    assert float(got[0].abs().max()) > 0
    assert torch.equal(got[0], got[1])
    st.free()


@pytest.mark.parametrize("explicit", [False, True])
def test_grid_calls_wait_for_the_default_stream(rt, explicit):
    from physis_gb300 import warmstart as ws
    shape = (9, 6, 5)
    st = ws.Stack([ws.make_instance(np.random.default_rng(6), shape)], shape, nsx=1)
    zc, yc, xc = ws.coarse_shape(shape, 4)
    f = st.fields(4)
    coarse = torch.randn(zc * yc * xc, generator=torch.Generator().manual_seed(7)).cuda()
    got = []
    for busy in (False, True):
        st.grids[1].copyin(np.zeros(st.gshape, np.float32))
        torch.cuda.synchronize()
        if busy:
            torch.cuda._sleep(BUSY)
        assert ps.lib().PSWarmStartUpsample(ctypes.byref(f), _p(coarse),
                                            ctypes.c_void_p(st.grids[1].dev_ptr),
                                            _handle(explicit)) == 0
        if not busy:
            torch.cuda.synchronize()
        got.append(st.grids[1].copyout())
    assert np.abs(got[0]).max() > 0
    assert np.array_equal(got[0], got[1])
    st.free()


def test_work_on_the_stream_given_out(rt):
    # what a program puts on PSGetStream's stream itself is ordered as well
    w, fwd = _weights(8)
    src, dw = w.cuda(), torch.zeros_like(w, device="cuda")
    wf, wb = torch.zeros_like(fwd, device="cuda"), torch.zeros_like(fwd, device="cuda")
    out = torch.zeros_like(wf)
    ext = torch.cuda.ExternalStream(ps.lib().PSGetStream())
    torch.cuda.synchronize()
    with torch.cuda.stream(ext):
        torch.cuda._sleep(BUSY)
        dw.copy_(src)
    assert ps.lib().PSWarmStartPrepareWeights(_p(dw), _p(wf), _p(wb), None) == 0
    with torch.cuda.stream(ext):
        out.copy_(wf)
    ext.synchronize()
    assert torch.equal(out.cpu(), fwd)
