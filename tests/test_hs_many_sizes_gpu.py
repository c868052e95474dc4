"""A Horn-Schunck batch of more frame sizes than a context keeps plans for: the
first plans are dropped before the call ends, and the flows are those of single
solves."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("device", [False, True])
def test_more_sizes_than_plans(of, device):
    import torch
    from oflow import synth
    prm = of.HSParams(15.0, 1, 1, 10)
    pairs = []
    for k in range(20):
        q = synth.hs_pair(seed=k, w=40 + 3 * k, h=32 + k)
        pairs.append((q.I0, q.I1))
    c = of.Context(0)
    given = [tuple(torch.from_numpy(x).cuda() for x in p) for p in pairs] if device else pairs
    for _ in range(2):
        res = of.hs_batch(given, prm, c)
        for (a, b), (u, v) in zip(pairs, res):
            if device:
                u, v = u.cpu().numpy(), v.cpu().numpy()
            su, sv = of.hs(a, b, prm)
            assert np.array_equal(u, su) and np.array_equal(v, sv)
    c.close()
