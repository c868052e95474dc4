"""Objects made while the default stream is busy: what their constructors clear
and copy is there before a stream that does not wait for the default one uses
it."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _busy():
    import torch
    torch.cuda.synchronize()
    torch.cuda._sleep(400_000_000)  # about 0.2 s


@pytest.fixture
def own_stream(of):
    import torch
    s = torch.cuda.Stream()  # does not wait for the default stream
    c = of.Context(0)
    c.set_stream(s.cuda_stream)
    yield c, s
    torch.cuda.synchronize()
    c.close()


def test_network_parameters(of, own_stream):
    import torch
    from oflow import warmstart
    c, s = own_stream
    params = warmstart.load()[0]
    frames = torch.randint(0, 256, (1, 2, 48, 64), dtype=torch.uint8, device="cuda")
    nets = []
    for busy in (False, True):
        if busy:
            _busy()
        net = of.WarmNet(64, 48, 1, c)
        net.set_params(params)
        nets.append((net, net.predict(frames)))
    torch.cuda.synchronize()
    assert np.array_equal(nets[1][0].get_params(), np.asarray(params, np.float32).ravel())
    assert torch.equal(nets[0][1], nets[1][1])
    # the packed weights too, once everything has landed
    first, second = (n.predict(frames) for n, _ in nets)
    torch.cuda.synchronize()
    assert torch.equal(first, second)


def test_tvl1_plan_and_stream(of, own_stream):
    import torch
    from oflow import synth
    c, s = own_stream
    prm = of.TVL1Params(nscales=3, max_iterations=8)
    p = synth.tvl1_pair(seed=5, w=96, h=64, radius=12)
    a, b = (torch.from_numpy(synth.quantize(x)).cuda() for x in (p.I0, p.I1))
    zero = torch.zeros_like(a)
    want = of.tvl1(a.cpu().numpy(), b.cpu().numpy(), prm)
    want0 = of.tvl1(zero.cpu().numpy(), a.cpu().numpy(), prm)
    got, got0 = (tuple(torch.empty((64, 96), device="cuda") for _ in range(2)) for _ in range(2))
    _busy()
    of.tvl1_batch([(a, b)], prm, c, out=[got])
    _busy()
    st = of.FrameStream(96, 64, "tvl1", 1, prm, "u8", c)
    st.push([a], out=[got0])
    torch.cuda.synchronize()
    st.close()
    for g, r in ((got, want), (got0, want0)):
        assert all(np.array_equal(x.cpu().numpy(), y) for x, y in zip(g, r))
