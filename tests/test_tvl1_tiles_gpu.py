"""The tiled TV-L1 iterations, whose state lives in registers, against the
oracle: every tile shape at the sizes where its edges, remainders and border
forms meet, and the inputs that break the fast arithmetic's guard (the tile is
then run again with every branch).  The kernels perform the oracle's operations
with the oracle's roundings, so the flows and iteration counts are equal."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _same(of, orc, ctx, a, b, prm):
    u, v, st = of.tvl1(a, b, prm, ctx, stats=True)
    ou, ov, its, _ = orc.tvl1(a.astype(np.float32), b.astype(np.float32),
                              orc.TVL1Params(prm.tau, prm.lambda_, prm.theta, prm.nscales, prm.zfactor,
                                             prm.warps, prm.epsilon, prm.max_iterations),
                              error_mode=1, trace=True)
    assert np.array_equal(st["iterations"], its)
    assert np.array_equal(u, ou) and np.array_equal(v, ov)


# owned tiles are 56 wide and 40, 24, 16, 8 high, regions 64 wide; odd widths
# have no aligned pixel pairs
@pytest.mark.parametrize("cfg", range(4))
@pytest.mark.parametrize("w,h", [(14, 9), (55, 41), (56, 40), (57, 16), (64, 24), (113, 25), (170, 81), (171, 49)])
def test_tile_edges(of, orc, monkeypatch, cfg, w, h):
    from oflow import synth
    monkeypatch.setenv("OFLOW_TB_CFG", str(cfg))
    p = synth.tvl1_pair(seed=w * 31 + h, w=w, h=h, radius=min(w, h) / 4.0)
    _same(of, orc, of.Context(0), synth.quantize(p.I0), synth.quantize(p.I1),
          of.TVL1Params(nscales=1, warps=2, max_iterations=11))


# the resident form: columns and rows per thread, blocks per cluster; widths of
# one to three warps, bands with empty rows, a last block without any
@pytest.mark.parametrize("form", ["1,1,1", "1,1,2", "1,1,16", "2,1,1", "2,1,4", "2,1,16", "2,2,1", "2,2,8", "2,2,16"])
@pytest.mark.parametrize("w,h", [(14, 9), (31, 15), (33, 16), (64, 15), (65, 17), (97, 31), (130, 33), (161, 62)])
def test_resident_level(of, orc, monkeypatch, form, w, h):
    from oflow import synth
    monkeypatch.setenv("OFLOW_TB_CFG", "5")
    monkeypatch.setenv("OFLOW_RES", form)
    p = synth.tvl1_pair(seed=w * 37 + h, w=w, h=h, radius=min(w, h) / 4.0)
    c = of.Context(0)
    for mi in (0, 1, 23):
        _same(of, orc, c, synth.quantize(p.I0), synth.quantize(p.I1),
              of.TVL1Params(nscales=1, warps=2, max_iterations=mi))


@pytest.mark.parametrize("cfg", ["0", "5"])
@pytest.mark.parametrize("case", ["steep", "tiny", "static"])
def test_guard(of, orc, monkeypatch, case, cfg):
    """steep: frames that are not normalised (their range is negative), with
    |grad|^2 above 2^24; tiny: steps so small that numerators of the dual
    update fall below 2^-100; static: equal frames, all numerators zero."""
    from oflow import synth
    monkeypatch.setenv("OFLOW_TB_CFG", cfg)
    p = synth.tvl1_pair(seed=9, w=130, h=90, radius=20)
    a, b = p.I0.astype(np.float32), p.I1.astype(np.float32)
    prm = of.TVL1Params(nscales=1, warps=2, max_iterations=9, epsilon=0.0)
    if case == "steep":
        a, b = -1000.0 - 300.0 * a, -1000.0 - 300.0 * b
    elif case == "tiny":
        prm.lambda_ = 1e-33
    else:
        b = a
    _same(of, orc, of.Context(0), a, b, prm)
