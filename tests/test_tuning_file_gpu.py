"""Saved tuning tables say which shape a number stands for.  A table without
shapes, or with others, was tuned among other kernels: it loads, and its numbers
are left out.  (Saving a context's table again shows what was taken.)"""
import pytest

pytestmark = pytest.mark.gpu


def _taken(of, tmp_path, text):
    a, b = tmp_path / "a.txt", tmp_path / "b.txt"
    a.write_text(text)
    c = of.Context(0)
    c.load_tuning(str(a))
    c.save_tuning(str(b))
    c.close()
    return sorted(l.strip() for l in open(b) if not l.startswith("#"))


def test_old_and_new_tables(of, tmp_path):
    old = "# oflow tuning table: solver level_width level_height batch config\nhs 320 240 64 5\ntvl1 1024 436 32 0\n"
    assert _taken(of, tmp_path, old) == []
    new = ["hs 320 240 64 2 48x48/8", "hs 160 120 1 5 48x16/8", "tvl1 1024 436 32 0 56x40", "tvl1 64 28 32 4 block",
           "tvl1 128 55 32 5 cluster"]
    assert _taken(of, tmp_path, "\n".join(new) + "\n") == sorted(new)
    other = ["hs 320 240 64 2 64x32/8", "tvl1 1024 436 32 0 64x32", "hs 320 240 64 9 48x48/8", "tvl1 64 28 32 6 cluster"]
    assert _taken(of, tmp_path, "\n".join(other) + "\n") == []


def test_malformed_lines_are_refused(of, tmp_path):
    c = of.Context(0)
    for text in ("tvl1 1 2\n", "hs 320 240 64 -1 48x48/8\n"):
        p = tmp_path / "bad.txt"
        p.write_text(text)
        with pytest.raises(of.OflowError):
            c.load_tuning(str(p))
    c.close()


def test_every_configuration_is_named(of, tmp_path):
    """What the autotuner picks comes back from a saved table."""
    from oflow import synth
    q = synth.hs_pair(seed=7, w=96, h=64)
    a, b, c = tmp_path / "a.txt", tmp_path / "b.txt", of.Context(0)
    of.hs_autotune([(q.I0, q.I1)], of.HSParams(15.0, 2, 1, 16), c)
    p = synth.tvl1_pair(seed=7, w=96, h=64, radius=12)
    of.tvl1_autotune([(synth.quantize(p.I0), synth.quantize(p.I1))], of.TVL1Params(nscales=2, max_iterations=8), c)
    c.save_tuning(str(a))
    c.close()
    lines = sorted(l.strip() for l in open(a) if not l.startswith("#"))
    assert len(lines) == 4 and all(len(l.split()) == 6 for l in lines)
    assert _taken(of, tmp_path, open(a).read()) == lines
