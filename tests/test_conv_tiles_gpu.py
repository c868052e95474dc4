"""The tcgen05 forward convolution and its backward-data form hold an input
region in shared memory and offset the matrix descriptors by taps: tile edges
and remainders in every mode and tile width, K padded to 16, channels that come
in several regions, weight stages of every depth, against the float64 oracle.
The products of bf16 operands are exact in float32; the sums of at most 9 C
terms in float32 stay within 9 C 2^-24 of the sum of magnitudes, which is some
sqrt(9 C) times the largest result: 2e-3 of it holds for every C here."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
REL = 2e-3


def _rel(a, b):
    return float(np.abs(a - b).max() / max(np.abs(b).max(), 1e-12))


@pytest.mark.parametrize("N,H,W,C,K,stride", [
    (1, 1, 1, 16, 16, 1), (1, 16, 8, 32, 8, 1), (2, 17, 9, 64, 48, 1), (1, 33, 31, 48, 128, 1),   # one accumulator
    (60, 31, 47, 32, 64, 1), (60, 33, 63, 160, 32, 1), (60, 32, 65, 16, 128, 1),                   # two and four
    (1, 2, 2, 16, 32, 2), (1, 32, 16, 96, 96, 2), (2, 35, 33, 96, 64, 2), (60, 65, 63, 32, 16, 2),
    (1, 20, 19, 512, 32, 1), (1, 34, 18, 512, 16, 2), (1, 18, 10, 768, 128, 1),                   # several regions
])
def test_forward_and_backward_data(of, N, H, W, C, K, stride):
    import torch
    from oracle import cnn_ref
    g = torch.Generator().manual_seed(H * 100 + W + C)
    P, Q = cnn_ref.conv_out(H, stride), cnn_ref.conv_out(W, stride)
    m = min(N, 2)  # the images of a batch repeat
    x = torch.randn((m, H, W, C), generator=g).bfloat16()
    w = (torch.randn((K, 3, 3, C), generator=g) * 0.1).bfloat16()
    b = torch.randn(K, generator=g) * 0.1
    rep = lambda t: t.repeat(N // m, 1, 1, 1).cuda().contiguous()
    ref = cnn_ref.forward(x.float().numpy(), w.float().numpy(), b.numpy(), stride, True)
    for f32 in (True, False):
        y = torch.full((N, P, Q, K), float("nan"), dtype=torch.float32 if f32 else torch.bfloat16, device="cuda")
        of.conv3x3(0, N, H, W, C, K, stride, True, f32, rep(x), None, w.cuda(), y, bias=b.cuda())
        got = y.float().cpu().numpy()
        assert all(_rel(got[i:i + m], ref) < (REL if f32 else 1e-2) for i in range(0, N, m))
    gout = torch.randn((m, P, Q, K), generator=g).bfloat16().float()
    gx_ref = cnn_ref.backward(x.float().numpy(), w.float().numpy(), gout.numpy(), stride, None)[0]
    gx = torch.full((N, H, W, C), float("nan"), dtype=torch.float32, device="cuda")
    of.conv3x3(1, N, H, W, C, K, stride, False, True, rep(gout), None, w.cuda(), gx)
    got = gx.cpu().numpy()
    assert all(_rel(got[i:i + m], gx_ref) < REL for i in range(0, N, m))


@pytest.mark.parametrize("N,H,W,C,K,stride", [
    (1, 1, 1, 16, 8, 1), (1, 16, 8, 32, 16, 1), (2, 17, 9, 48, 48, 1), (3, 31, 15, 80, 128, 1), (2, 50, 70, 96, 80, 1),
    (1, 2, 2, 16, 32, 2), (2, 33, 17, 32, 96, 2), (1, 64, 31, 208, 112, 2), (40, 47, 33, 16, 24, 1),
])
def test_backward_weight(of, N, H, W, C, K, stride):
    """Channel groups of every remainder (up to five a block), pixel tiles with
    remainders, one tile and several a block, K padded to 16."""
    import torch
    from oracle import cnn_ref
    g = torch.Generator().manual_seed(H * 100 + W + C + 1)
    P, Q = cnn_ref.conv_out(H, stride), cnn_ref.conv_out(W, stride)
    x = torch.randn((N, H, W, C), generator=g).bfloat16()
    gout = torch.randn((N, P, Q, K), generator=g).bfloat16().float()
    w = torch.zeros((K, 3, 3, C)).bfloat16()
    gw_ref = cnn_ref.backward(x.float().numpy(), w.float().numpy(), gout.numpy(), stride, None)[1]
    gw = torch.full((K, 3, 3, C), float("nan"), dtype=torch.float32, device="cuda")
    gb = torch.empty(K, dtype=torch.float32, device="cuda")
    of.conv3x3(2, N, H, W, C, K, stride, False, True, gout.cuda(), None, x.cuda(), gw, gbias=gb)
    torch.cuda.synchronize()
    # gw is [K][3][3][C]; float32 sums of N P Q exact products
    assert _rel(gw.cpu().numpy(), gw_ref) < REL
