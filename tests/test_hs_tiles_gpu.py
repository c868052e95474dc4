"""The Horn-Schunck Jacobi tiles, whose state lives in registers, against the
oracle: every configuration at even sizes (regions by TMA) and odd ones where
tile edges, remainders and border forms meet, several tiles a block, and the
inputs that break the division's guard (the tile is then run again with IEEE
divisions).  Same operations and roundings, so the flows are equal."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("cfg", range(6))
@pytest.mark.parametrize("w,h,sweeps", [(6, 3, 5), (48, 16, 16), (50, 17, 9), (56, 57, 8), (112, 49, 21), (145, 33, 16)])
def test_tile_edges(of, orc, monkeypatch, cfg, w, h, sweeps):
    from oflow import synth
    monkeypatch.setenv("OFLOW_HS_CFG", str(cfg))
    c = of.Context(0)
    qs = [synth.hs_pair(seed=w + h + k, w=w, h=h) for k in range(2)]
    res = of.hs_batch([(q.I0, q.I1) for q in qs], of.HSParams(4.0, 1, 1, sweeps), c)
    c.close()
    for q, (u, v) in zip(qs, res):
        ou, ov = orc.hs(q.I0, q.I1, 4.0, 1, 1, sweeps)
        assert np.array_equal(u, ou) and np.array_equal(v, ov)


def test_several_tiles_per_block(of, orc):
    """More tiles than resident blocks, so that blocks fetch ahead."""
    from oflow import synth
    q = synth.hs_pair(seed=3, w=320, h=240)
    c = of.Context(0)
    res = of.hs_batch([(q.I0, q.I1)] * 12, of.HSParams(15.0, 1, 1, 20), c)
    c.close()
    ou, ov = orc.hs(q.I0, q.I1, 15.0, 1, 1, 20)
    assert all(np.array_equal(u, ou) and np.array_equal(v, ov) for u, v in res)


@pytest.mark.parametrize("n", [1, 3])
@pytest.mark.parametrize("sweeps", [1, 4, 7, 8, 9, 24])
@pytest.mark.parametrize("w,h", [(1, 1), (48, 128), (49, 65), (192, 64), (193, 63), (224, 96), (113, 169), (57, 361),
                                 (225, 97), (784, 10)])
def test_resident_levels(of, orc, w, h, sweeps, n):
    """Levels of one and of several blocks of a cluster, up to 16 of 48x16 (8
    sweeps between exchanges) and of 56x24 (4), and the first ones beyond."""
    from oflow import synth
    qs = [synth.hs_pair(seed=w + h + k, w=w, h=h) for k in range(n)]
    c = of.Context(0)
    res = of.hs_batch([(q.I0, q.I1) for q in qs], of.HSParams(4.0, 1, 2, sweeps), c)
    c.close()
    for q, (u, v) in zip(qs, res):
        ou, ov = orc.hs(q.I0, q.I1, 4.0, 1, 2, sweeps)
        assert np.array_equal(u, ou) and np.array_equal(v, ov)


@pytest.mark.parametrize("w,h", [(130, 70), (131, 45), (200, 90)])
@pytest.mark.parametrize("scale,alpha", [(1e-32, 1.0), (1e4, 1.0), (0.0, 1e-14)])
def test_resident_guard(of, orc, scale, alpha, w, h):
    """One pair: the whole cluster runs the warp again with IEEE divisions."""
    from oflow import synth
    q = synth.hs_pair(seed=11, w=w, h=h)
    a, b = (q.I0 * scale).astype(np.float32), (q.I1 * scale).astype(np.float32)
    c = of.Context(0)
    u, v = of.hs(a, b, of.HSParams(alpha, 1, 1, 19), c)
    c.close()
    ou, ov = orc.hs(a, b, alpha, 1, 1, 19)
    assert np.array_equal(u, ou) and np.array_equal(v, ov)


@pytest.mark.parametrize("w", [130, 131])
@pytest.mark.parametrize("scale,alpha", [(1e-32, 1.0), (1e4, 1.0), (0.0, 1e-14)])
def test_guard(of, orc, scale, alpha, w):
    """Numerators below 2^-100, denominators above 2^24 and below 2^-40."""
    from oflow import synth
    q = synth.hs_pair(seed=11, w=w, h=70)
    a, b = (q.I0 * scale).astype(np.float32), (q.I1 * scale).astype(np.float32)
    c = of.Context(0)
    res = of.hs_batch([(a, b)] * 16, of.HSParams(alpha, 1, 1, 19), c)
    c.close()
    ou, ov = orc.hs(a, b, alpha, 1, 1, 19)
    assert all(np.array_equal(u, ou) and np.array_equal(v, ov) for u, v in res)
