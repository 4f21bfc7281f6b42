"""The warm-start network's tiled kernels at the sizes where they can go
wrong: fewer voxels than a tile, tile and part edges, one-cell axes, rows
longer than a tile, more splits than voxels, and rows too long to stage."""
import ctypes

import numpy as np
import pytest

import physis_gb300 as ps
from oracle import nn_oracle as nn

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


@pytest.fixture(scope="module")
def rt():
    ps.build()
    ps.init()
    yield ps
    ps.clear_error()


def _bf(a):
    return torch.tensor(nn.to_bf16(a).view(np.int16).ravel(), device="cuda").view(torch.bfloat16)


def _p(t):
    return ctypes.c_void_p(t.data_ptr())


def _stream():
    # PyTorch's default stream is handle 0, which the library takes for its own
    # stream; 1 is CUDA's name for the default stream (cudaStreamLegacy)
    return ctypes.c_void_p(torch.cuda.current_stream().cuda_stream or 1)


# FP32 sums of n products of O(1) BF16 values, added in runs of 16 (a tensor
# instruction) and in trees of parts: the error of each of the at most n / 16
# sequential additions is 2^-24 of a partial sum of about sqrt(n), so it stays
# below sqrt(n / 16) * 2^-24 * sqrt(n) < 4e-5 for the 10^4 voxels used here,
# under 1e-5 of the largest gradient (about 3 sqrt(n)).
@pytest.mark.parametrize("dims,nsplit", [
    ((1, 1, 1, 1), 1), ((1, 1, 1, 1), 5), ((1, 1, 1, 16), 2), ((1, 1, 3, 85), 1),
    ((1, 2, 2, 64), 1), ((1, 1, 1, 257), 1), ((2, 3, 1, 300), 3), ((1, 7, 11, 13), 64),
    ((5, 2, 3, 1), 2), ((3, 4, 1, 1), 1), ((4, 17, 9, 9), 7), ((1, 1, 2, 1300), 2),
    ((1, 3, 31, 31), 2), ((1, 2, 33, 31), 1), ((2, 2, 40, 41), 3), ((40, 17, 9, 9), 64)])
def test_weight_gradient_edges(rt, dims, nsplit):
    rng = np.random.default_rng(31)
    x = nn.from_bf16(nn.to_bf16(rng.normal(size=dims + (16,))))
    dy = nn.from_bf16(nn.to_bf16(rng.normal(size=dims + (16,))))
    work = torch.full((nsplit * (27 * 256 + 16),), float("nan"), device="cuda")
    dw = torch.empty(27 * 256, dtype=torch.float32, device="cuda")
    db = torch.empty(16, dtype=torch.float32, device="cuda")
    tx, tdy = _bf(x), _bf(dy)
    rc = ps.lib().PSWarmStartWeightGrad(_p(tx), _p(tdy), _p(work), nsplit, _p(dw), _p(db),
                                        *dims, _stream())
    assert rc == 0
    rdw, rdb = nn.conv_bwd_weight(x, dy)
    got = dw.cpu().numpy().reshape(27, 16, 16)
    assert np.abs(got - rdw).max() <= 1e-5 * max(np.abs(rdw).max(), 1.0)
    assert np.abs(db.cpu().numpy() - rdb).max() <= 1e-5 * max(np.abs(rdb).max(), 1.0)


# The padded-slab convolution: slabs of one and of several planes, planes of
# one voxel, up to and past the 1024 padded voxels a slab may have, rows and
# columns past the 256-voxel box.  BF16 outputs within one rounding step of the
# FP64 value plus the FP32 error of 432 products of O(1) values (432 * 2^-24).
@pytest.mark.parametrize("dims", [
    (1, 1, 1, 1), (1, 2, 1, 1), (2, 1, 1, 127), (1, 1, 63, 1), (1, 3, 7, 15), (1, 5, 31, 31),
    (1, 2, 32, 31), (1, 1, 3, 255), (1, 2, 2, 256), (1, 1, 256, 2), (700, 3, 4, 4),
    (3, 40, 5, 6)])
@pytest.mark.parametrize("masked", [False, True])
def test_conv_edges(rt, dims, masked):
    rng = np.random.default_rng(32)
    x = nn.from_bf16(nn.to_bf16(rng.normal(size=dims + (16,))))
    m = nn.from_bf16(nn.to_bf16(rng.normal(size=dims + (16,))))
    w = nn.from_bf16(nn.to_bf16(rng.normal(0, 0.2, size=(27, 16, 16)))).astype(np.float32)
    bias = rng.normal(0, 0.1, 16).astype(np.float32)
    wt = torch.tensor(w.ravel(), device="cuda")
    wf = torch.empty(27 * 256, dtype=torch.bfloat16, device="cuda")
    wb = torch.empty(27 * 256, dtype=torch.bfloat16, device="cuda")
    assert ps.lib().PSWarmStartPrepareWeights(_p(wt), _p(wf), _p(wb), _stream()) == 0
    n = int(np.prod(dims))
    y = torch.full((n * 16,), float("nan"), dtype=torch.bfloat16, device="cuda")
    y0 = torch.empty(n, dtype=torch.float32, device="cuda")
    tx, tm, tb = _bf(x), _bf(m), torch.tensor(bias, device="cuda")
    if masked:  # the backward-data form
        rc = ps.lib().PSWarmStartConv(_p(tx), _p(wb), None, _p(tm), 0, _p(y), None, *dims,
                                      _stream())
        ref = nn.conv_bwd_data(x, w) * (m > 0)
    else:
        rc = ps.lib().PSWarmStartConv(_p(tx), _p(wf), _p(tb), None, 1, _p(y), _p(y0), *dims,
                                      _stream())
        ref = nn.relu(nn.conv_fwd(x, w, bias))
    assert rc == 0
    got = nn.from_bf16(y.view(torch.int16).cpu().numpy().view(np.uint16)).reshape(dims + (16,))
    tol = np.abs(ref) * 2.0 ** -7 + 3e-5 * np.abs(ref).max() + 1e-30
    assert np.all(np.abs(got - ref) <= tol)
    if not masked:
        assert np.allclose(y0.cpu().numpy().reshape(dims), ref[..., 0], rtol=3e-5,
                           atol=3e-5 * np.abs(ref).max())


# One launch over the whole network against the per-layer calls it replaces:
# the same arithmetic, so the same weights, moments and BF16 copies up to one
# FP32 rounding (contraction may differ between the kernels): 2^-23 relative
# on the moments, the update itself being at most lr.
@pytest.mark.parametrize("layers", [1, 3, 6])
def test_adam_layers_matches_single_calls(rt, layers):
    L = ps.lib()
    per, n = 27 * 256, layers * (27 * 256 + 16)
    gen = torch.Generator(device="cuda").manual_seed(5)
    w, g, m = (torch.randn(n, generator=gen, device="cuda") for _ in range(3))
    v = torch.rand(n, generator=gen, device="cuda")
    w2, m2, v2 = w.clone(), m.clone(), v.clone()
    half = torch.zeros((2, layers, per), dtype=torch.bfloat16, device="cuda")
    half2 = torch.zeros_like(half)
    assert L.PSWarmStartAdamLayers(_p(w), _p(g), _p(m), _p(v), layers, 1e-2, 0.9, 0.999, 1e-8, 3,
                                   _p(half[0]), _p(half[1]), _stream()) == 0
    assert L.PSWarmStartAdam(_p(w2), _p(g), _p(m2), _p(v2), n, 1e-2, 0.9, 0.999, 1e-8, 3,
                             _stream()) == 0
    for l in range(layers):
        assert L.PSWarmStartPrepareWeights(_p(w[l * per:]), _p(half2[0, l]), _p(half2[1, l]),
                                           _stream()) == 0
    torch.cuda.synchronize()
    assert torch.allclose(m, m2, rtol=2 ** -23, atol=0) and torch.allclose(v, v2, rtol=2 ** -23,
                                                                           atol=0)
    assert (w - w2).abs().max() <= 2 ** -22 * w2.abs().max()
    assert torch.equal(half.view(torch.int16), half2.view(torch.int16))


@pytest.mark.parametrize("batch", [16, 47])
def test_loss_is_that_of_its_own_prediction(rt, batch):
    # the host reads the loss right after the kernels were issued, on PyTorch's
    # default stream: it must be this step's, step after step
    from physis_gb300 import warmstart as ws
    dims = (batch, 16, 16, 16)
    gen = torch.Generator(device="cuda").manual_seed(6)
    n = int(np.prod(dims))
    x = torch.randn(n * 16, generator=gen, device="cuda").to(torch.bfloat16)
    t = torch.randn(n, generator=gen, device="cuda")
    net = ws.Net(7)
    work = torch.empty(64 * (27 * 256 + 16), device="cuda")
    work64 = torch.empty((n + 255) // 256, dtype=torch.float64, device="cuda")
    for _ in range(4):
        pred = net.forward(x, dims)
        loss, dy = ws.loss_grad(pred, t, work64)
        net.backward(dy, dims, work)
        net.adam(2e-3)
        true = float(((pred - t).double() ** 2).mean())  # FP32 difference, as the kernel's
        assert abs(loss - true) <= 1e-9 * true


@pytest.mark.parametrize("side", [False, True])
def test_overlapping_launches_keep_their_order(rt, monkeypatch, side):
    # every launch of a step may start as the one before it ends; in turn
    # (PS_OVERLAP=0) gives the same bits, on PyTorch's stream and on another
    from physis_gb300 import warmstart as ws
    dims = (9, 17, 9, 9)
    n = int(np.prod(dims))
    gen = torch.Generator(device="cuda").manual_seed(8)
    x = torch.randn(n * 16, generator=gen, device="cuda").to(torch.bfloat16)
    t = torch.randn(n, generator=gen, device="cuda")
    torch.cuda.synchronize()
    got = []
    for env in ("0", "1", "1"):
        monkeypatch.setenv("PS_OVERLAP", env)
        with torch.cuda.stream(torch.cuda.Stream() if side else torch.cuda.default_stream()):
            net = ws.Net(7)
            work = torch.empty(64 * (27 * 256 + 16), device="cuda")
            work64 = torch.empty((n + 255) // 256, dtype=torch.float64, device="cuda")
            losses = []
            for _ in range(6):
                loss, dy = ws.loss_grad(net.forward(x, dims), t, work64)
                net.backward(dy, dims, work)
                net.adam(2e-3)
                losses.append(float(loss))
            out = net.forward(x, dims).clone()
            torch.cuda.current_stream().synchronize()
        got.append((losses, out))
    for losses, out in got[1:]:
        assert losses == got[0][0]
        assert torch.equal(out, got[0][1])
