"""The replicas that long runs fold histories into (csrc/mc_event.cu,
single_replicas) keep to lines of their own: a problem of three bins costs no
more than the same one with bins that nothing scores."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

DECK = """<?xml version="1.0"?>
<simulation><description name="r" samples="100"/></simulation>
<multigroup groups="1"/>
<materials><material name="m"><multigroup total="1.0" scatter="0.5"/></material></materials>
<surfaces><plane_x name="a" x="0"/><plane_x name="b" x="3"/><plane_x name="c" x="4"/></surfaces>
<cells>
<cell name="slab" material="m" importance="1"><surface name="a" sense="+1"/><surface name="b" sense="-1"/></cell>
<cell name="left" importance="0"><surface name="a" sense="-1"/></cell>
<cell name="right" importance="0"><surface name="b" sense="+1"/><surface name="c" sense="-1"/></cell>
<cell name="far" material="m" importance="1"><surface name="c" sense="+1"/></cell>
</cells>
<distributions><delta name="e" datatype="double" val="1e6"/><delta name="d" datatype="point" x="1" y="0" z="0"/></distributions>
<sources><point x="0.001" y="0" z="0" direction="d" energy="e" group="0"/></sources>
<estimators><estimator name="s" type="C" scores="total capture scatter"><cell name="slab"/></estimator>%s</estimators>
"""
FAR = '<estimator name="f" type="C" scores="flux"><cell name="far"/><filter type="energy" grid_lethargy="1e-5 2e7 60"/></estimator>'


def _run(folder, extra):
    import mcgpu
    folder.mkdir()
    (folder / "input.xml").write_text(DECK % extra)
    p = mcgpu.Problem(str(folder))
    ms = []
    for r in range(9):
        p.reset()
        c = p.run(n=1_000_000, seed=5, mode="event", kernel=2)
        assert c["launches"] == 2
        ms.append(c["total_ms"])
    s = p.all_tallies()[2].copy()
    p.close()
    return min(ms[2:]), s


def test_three_bins_cost_no_more_than_with_bins_that_nothing_scores(tmp_path):
    ms, s = _run(tmp_path / "three", "")
    wide_ms, w = _run(tmp_path / "wide", FAR)
    assert len(s) == 3 and len(w) > 48 and np.all(s > 0) and not np.any(w[3:])
    # the same histories' terms in another order: n 2^-53 for a sum of nonnegative ones
    assert np.all(np.abs(s - w[:3]) <= 8e6 * 2.0 ** -53 * s)
    assert ms <= 1.25 * wide_ms, (ms, wide_ms)
