"""Two threads run layers of one kernel that take different amounts of shared
memory, on streams of their own: every call succeeds and gives the same result."""
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mode", [0, 2])
def test_layers_of_different_size_at_once(of, mode):
    import torch
    N, H, W, K = 1, 16, 16, 64
    g = torch.Generator().manual_seed(mode)
    start, failed = threading.Barrier(2), []

    def work(C):
        x = torch.randn((N, H, W, C), generator=g).bfloat16().cuda()
        other = (torch.randn((K, 3, 3, C), generator=g).bfloat16() if mode == 0 else torch.randn((N, H, W, K), generator=g)).cuda()
        b = torch.zeros(K, device="cuda")
        y = torch.empty((N, H, W, K) if mode == 0 else (K, 3, 3, C), dtype=torch.float32, device="cuda")
        torch.cuda.synchronize()
        start.wait()
        first = None
        for _ in range(400):
            try:
                if mode == 0:
                    of.conv3x3(0, N, H, W, C, K, 1, False, True, x, None, other, y, bias=b)
                else:
                    of.conv3x3(2, N, H, W, C, K, 1, False, True, other, None, x, y, gbias=b)
            except of.capi.OflowError as e:
                failed.append((C, str(e)))
                return
            first = y.cpu().numpy() if first is None else first
        torch.cuda.synchronize()
        # (one tile a channel group in mode 2 too: no order of additions to differ)
        if not np.allclose(y.cpu().numpy(), first, rtol=1e-5, atol=1e-4):
            failed.append((C, "another result"))

    threads = [threading.Thread(target=work, args=(C,)) for C in (16, 224)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not failed
