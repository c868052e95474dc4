"""A mixed batch kept from an earlier call serves jobs in another order: each
job gets its own frames' flow (oflow_batch groups jobs by solver, size, dtype
and parameters, and keeps the plans by the groups)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("device", [False, True])
def test_kept_batch_with_jobs_in_another_order(of, device):
    import torch
    from oflow import synth
    prm = of.HSParams(15.0, 1, 1, 12)
    jobs = []
    for k, (w, h) in enumerate([(48, 40), (48, 40), (64, 32)]):
        q = synth.hs_pair(seed=60 + k, w=w, h=h)
        f = (q.I0, q.I1)
        jobs.append(("hs",) + (tuple(torch.from_numpy(x).cuda() for x in f) if device else f) + (prm,))
    c = of.Context(0)

    def flows(order):
        res = of.batch([jobs[i] for i in order], c)
        return {i: [x.cpu().numpy() if device else x for x in uv] for i, uv in zip(order, res)}

    first = flows([0, 1, 2])
    for order in ([0, 2, 1], [1, 0, 2], [1, 2, 0]):
        for i, (u, v) in flows(order).items():
            assert np.array_equal(u, first[i][0]) and np.array_equal(v, first[i][1]), (order, i)
    c.close()
