"""Layers whose input channels come in several regions of the tcgen05 forward
kernel, with two weight buffers and enough blocks that the loader threads of a
block drift apart: every region waits for the products of the one before it.
Against the float64 oracle, many times; sums of 9 C exact products in float32
(the tolerance of the other tile tests)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
REL = 2e-3


def _rel(a, b):
    return float(np.abs(a - b).max() / max(np.abs(b).max(), 1e-12))


@pytest.mark.parametrize("mode,H,W,C,K,stride", [(0, 34, 26, 768, 128, 1), (0, 35, 27, 768, 128, 2), (1, 24, 17, 32, 768, 1),
                                                 (1, 33, 31, 16, 768, 2)])
def test_many_blocks_of_several_regions(of, mode, H, W, C, K, stride):
    import torch
    from oracle import cnn_ref
    N = 48
    g = torch.Generator().manual_seed(C + K + stride)
    P, Q = cnn_ref.conv_out(H, stride), cnn_ref.conv_out(W, stride)
    x = torch.randn((1, H, W, C), generator=g).bfloat16()
    w = (torch.randn((K, 3, 3, C), generator=g) * 0.1).bfloat16()
    rep = lambda t: t.repeat(N, 1, 1, 1).cuda().contiguous()
    if mode == 0:
        b = torch.randn(K, generator=g) * 0.1
        ref = cnn_ref.forward(x.float().numpy(), w.float().numpy(), b.numpy(), stride, False)
        a, bd, shape = rep(x), b.cuda(), (N, P, Q, K)
    else:
        gout = torch.randn((1, P, Q, K), generator=g).bfloat16().float()
        ref = cnn_ref.backward(x.float().numpy(), w.float().numpy(), gout.numpy(), stride, None)[0]
        a, bd, shape = rep(gout), None, (N, H, W, C)
    wd = w.cuda()
    first = None
    for _ in range(10):
        y = torch.full(shape, float("nan"), dtype=torch.float32, device="cuda")
        of.conv3x3(mode, N, H, W, C, K, stride, False, True, a, None, wd, y, bias=bd)
        got = y.cpu().numpy()
        if first is None:
            first = got
            assert all(_rel(got[i:i + 1], ref) < REL for i in range(N))
        else:
            assert np.array_equal(got, first)
