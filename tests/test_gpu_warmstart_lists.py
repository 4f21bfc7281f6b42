"""Net's lists of parameters, gradients and moments are a program's to fill:
the optimiser step uses the tensors that are in them."""
import pytest

import physis_gb300 as ps

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


@pytest.fixture(scope="module")
def rt():
    ps.build()
    ps.init()
    yield ps
    ps.clear_error()


@pytest.mark.parametrize("lists", [("grads",), ("m", "v"), ("params",), ("w", "params"), ("wf", "wb"),
                                   ("grads", "m", "v", "params", "w", "wf", "wb")])
@pytest.mark.parametrize("how", ["entry", "data"])
def test_step_uses_the_tensors_in_the_lists(rt, lists, how):
    from physis_gb300 import warmstart as ws
    nets = [ws.Net(3), ws.Net(3)]
    gen = torch.Generator(device="cuda").manual_seed(4)
    values = [torch.randn(t.shape, generator=gen, device="cuda") for t in nets[0].grads]
    for net in nets:
        for g, v in zip(net.grads, values):
            g.copy_(v)
        net.adam(1e-2)  # moments that are not zero
    own = nets[1]
    fresh = {}  # one tensor for one entry, also where two lists hold it
    for name in lists:
        entries = getattr(own, name)
        for i, t in enumerate(entries):
            if how == "data":
                t.data = t.data.clone()
            else:
                entries[i] = fresh.setdefault(t.data_ptr(), t.clone())
    for net in nets:
        for g, v in zip(net.grads, values):
            g.copy_(v.flip(0))
        net.adam(1e-2)
    torch.cuda.synchronize()
    for name in ("params", "grads", "m", "v"):
        for a, b in zip(getattr(nets[0], name), getattr(own, name)):
            assert torch.equal(a, b), name
    # the BF16 copies are those of w's tensors
    for l, w in enumerate(own.w):
        half = w.reshape(27, 16, 16).to(torch.bfloat16)
        assert torch.equal(own.wf[l].reshape(27, 16, 16), half.transpose(1, 2))
        assert torch.equal(own.wb[l].reshape(27, 16, 16), half.flip(0))
