"""Backward-data takes weights at any bf16 address (they are read one by one) and
gives the same result there; the forward product takes 16-byte aligned ones and
refuses others, before anything is written."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shift", [1, 3, 8])
@pytest.mark.parametrize("stride", [1, 2])
def test_weights_address(of, shift, stride):
    import torch
    from oracle import cnn_ref
    N, H, W, C, K = 1, 19, 14, 48, 24
    P, Q = cnn_ref.conv_out(H, stride), cnn_ref.conv_out(W, stride)
    g = torch.Generator().manual_seed(shift)
    w = (torch.randn((K, 3, 3, C), generator=g) * 0.1).bfloat16().cuda()
    room = torch.zeros(w.numel() + 16, dtype=torch.bfloat16, device="cuda")
    moved = room[shift:shift + w.numel()].view(w.shape)
    moved.copy_(w)
    gout = torch.randn((N, P, Q, K), generator=g).cuda()
    x = torch.randn((N, H, W, C), generator=g).bfloat16().cuda()
    b = torch.zeros(K, device="cuda")
    gx = [torch.full((N, H, W, C), float("nan"), device="cuda") for _ in range(2)]
    for wt, o in zip((w, moved), gx):
        of.conv3x3(1, N, H, W, C, K, stride, False, True, gout, None, wt, o)
    assert torch.equal(gx[0], gx[1]) and not torch.isnan(gx[0]).any()
    y = torch.full((N, P, Q, K), 7.0, device="cuda")
    if shift % 8:
        with pytest.raises(of.capi.OflowError):
            of.conv3x3(0, N, H, W, C, K, stride, False, True, x, None, moved, y, bias=b)
        assert bool((y == 7.0).all())
    else:
        of.conv3x3(0, N, H, W, C, K, stride, False, True, x, None, moved, y, bias=b)
        there = torch.full_like(y, float("nan"))
        of.conv3x3(0, N, H, W, C, K, stride, False, True, x, None, w, there, bias=b)
        assert torch.equal(y, there)
