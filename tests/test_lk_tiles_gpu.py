"""The Lucas-Kanade kernels solve several pixels a thread in 32 x 32 tiles:
every window and tap count at tile edges and remainders, in launches of few
tiles (one row a thread) and of many (four rows), device frames and flows with
a pitch, odd base addresses and flows that overlap a frame.  Same operations
and roundings as the oracle, so the flows are equal."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _frames(w, h, n, seed):
    from oflow import synth
    rng = np.random.default_rng(seed)
    base = synth.value_noise(rng, h, w)
    return [synth.quantize(base + rng.normal(0, 2, base.shape) + k) for k in range(n)]


@pytest.mark.parametrize("window", [1, 3, 5, 7, 9])
@pytest.mark.parametrize("spac,temp", [(1, 1), (3, 2), (5, 3), (7, 5), (9, 9)])
@pytest.mark.parametrize("w,h", [(9, 9), (10, 41), (32, 32), (33, 31), (65, 70), (1003, 610)])
def test_single_step(of, orc, ctx, window, spac, temp, w, h):
    fr = _frames(w, h, temp, w + h)
    u, v = of.lk(fr, 3, of.LKParams(spac, temp, window), ctx)
    ou, ov = orc.lk_ring(fr, 3, spac, temp, window)
    assert np.array_equal(u, ou) and np.array_equal(v, ov)


@pytest.mark.parametrize("w,h", [(61, 45), (1000, 620)])
@pytest.mark.parametrize("offset", [0, 1])
def test_single_step_device_in_place(of, ctx, w, h, offset):
    import torch
    fr = _frames(w, h, 5, w)
    prm = of.LKParams(5, 5, 7)
    ru, rv = of.lk(fr, 2, prm, ctx)
    dev = []
    for f in fr:
        d = torch.zeros(h * (w + 7) + offset, dtype=torch.uint8, device="cuda:0")[offset:].view(h, w + 7)[:, :w]
        d.copy_(torch.from_numpy(f))
        dev.append(d)
    out = [torch.full((h, w + 3), 7.0, device="cuda:0") for _ in range(2)]
    torch.cuda.synchronize()
    of.lk(dev, 2, prm, ctx, out=(out[0][:, :w], out[1][:, :w]))
    torch.cuda.synchronize()
    for o, r in zip(out, (ru, rv)):
        assert np.array_equal(o[:, :w].cpu().numpy(), r) and torch.all(o[:, w:] == 7.0)
    # the frames in the memory that takes the flow
    both = torch.zeros((2, h, w), device="cuda:0")
    held = both.view(torch.uint8).view(-1)[: 5 * h * w].view(5, h, w)
    held.copy_(torch.from_numpy(np.stack(fr)))
    torch.cuda.synchronize()
    of.lk([held[k] for k in range(5)], 2, prm, ctx, out=(both[0], both[1]))
    torch.cuda.synchronize()
    assert np.array_equal(both[0].cpu().numpy(), ru) and np.array_equal(both[1].cpu().numpy(), rv)


@pytest.mark.parametrize("window", [1, 3, 5, 7, 9])
@pytest.mark.parametrize("spac", [1, 3, 5, 7, 9])
@pytest.mark.parametrize("w,h,n", [(31, 33, 2), (130, 67, 3), (64, 36, 200), (132, 70, 61)])
def test_pyramidal(of, orc, ctx, window, spac, w, h, n):
    """n copies of one pair: few tiles a launch and more than 592."""
    from oflow import synth
    l = synth.lk_pair(seed=w + h, w=w, h=h)
    res = of.pyrlk_batch([(l.I0, l.I1)] * n, of.LKParams(spac, 2, window, 2, 2), ctx)
    ou, ov = orc.pyrlk(l.I0, l.I1, 2, 2, spac, window)
    assert all(np.array_equal(u, ou) and np.array_equal(v, ov) for u, v in res)


def test_pyramidal_without_refinement(of, ctx):
    from oflow import synth
    l = synth.lk_pair(seed=3, w=40, h=36)
    u, v = of.pyrlk(l.I0, l.I1, of.LKParams(3, 2, 5, 2, 0), ctx)
    assert not u.any() and not v.any()
