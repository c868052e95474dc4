"""Horn-Schunck tiles fetched ahead without TMA (odd widths, and even ones in the
entry point that does not allocate, which has no flag for a bounded wait):
several tiles a block in every configuration, and tiles that run again while the
next one's data is on its way.  Flows equal the oracle's."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("cfg", range(6))
@pytest.mark.parametrize("still", [False, True])
def test_odd_widths(of, orc, monkeypatch, cfg, still):
    from oflow import synth
    monkeypatch.setenv("OFLOW_HS_CFG", str(cfg))
    w, h, n = 259, 129, 24  # 24 * 18 tiles of 48x48, and more of the others
    q = synth.hs_pair(seed=3, w=w, h=h)
    a, b = q.I0.astype(np.float32), q.I1.astype(np.float32)
    if still:
        y, x = np.mgrid[0:h, 0:w]
        disc = (x - 80) ** 2 + (y - 70) ** 2 < 200
        b = np.where(disc, np.roll(a, (1, 2), (0, 1)), a)
    sweeps = 130 if still else 21
    c = of.Context(0)
    res = of.hs_batch([(a, b)] * n, of.HSParams(4.0, 1, 1, sweeps), c)
    c.close()
    ou, ov = orc.hs(a, b, 4.0, 1, 1, sweeps)
    assert all(np.array_equal(u, ou) and np.array_equal(v, ov) for u, v in res)


@pytest.mark.parametrize("cfg", range(6))
@pytest.mark.parametrize("w,h", [(400, 300), (399, 301), (1, 400), (7, 3)])
def test_without_allocation(of, orc, monkeypatch, cfg, w, h):
    import torch
    from oflow import synth
    monkeypatch.setenv("OFLOW_HS_CFG", str(cfg))
    q = synth.hs_pair(seed=4, w=w, h=h)
    prm = of.HSParams(4.0, 1, 1, 37)
    I0, I1 = (torch.from_numpy(x.astype(np.float32)).cuda() for x in (q.I0, q.I1))
    u, v = (torch.full((h, w), float("nan"), device="cuda") for _ in range(2))
    torch.cuda.synchronize()
    p = prm.c()
    assert of.capi.lib().oflow_hs_noalloc(C.c_void_p(I0.data_ptr()), C.c_void_p(I1.data_ptr()), w, h, 0, C.byref(p),
                                          C.c_void_p(u.data_ptr()), C.c_void_p(v.data_ptr()), 0, C.c_void_p(0)) == 0
    torch.cuda.synchronize()
    ou, ov = orc.hs(q.I0, q.I1, 4.0, 1, 1, 37)
    assert np.array_equal(u.cpu().numpy(), ou) and np.array_equal(v.cpu().numpy(), ov)


def test_odd_widths_take_about_as_long(of):
    """641x479 has the tiles of 640x480; copies by cp.async instead of TMA cost
    instructions, not the wait for each tile's data (which doubled the time)."""
    import torch
    from oflow import synth
    st = torch.cuda.Stream()
    c = of.Context(0)
    c.set_stream(st.cuda_stream)
    prm = of.HSParams(1.0, 1, 1, 104)
    best = []
    for w, h in ((640, 480), (641, 479)):
        q = synth.hs_pair(seed=1, w=w, h=h)
        pairs = [tuple(torch.from_numpy(x.astype(np.float32)).cuda() for x in (q.I0, q.I1))] * 13
        out = [tuple(torch.empty((h, w), device="cuda") for _ in range(2)) for _ in range(13)]
        e = [torch.cuda.Event(enable_timing=True) for _ in range(2)]
        times = []
        for _ in range(8):
            torch.cuda.synchronize()
            e[0].record(st)
            of.hs_batch(pairs, prm, c, out=out)
            e[1].record(st)
            torch.cuda.synchronize()
            times.append(e[0].elapsed_time(e[1]))
        best.append(min(times[2:]))
    c.close()
    assert best[1] < 1.6 * best[0], best
