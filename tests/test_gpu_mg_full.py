"""Multigroup problems with a time filter, two filters besides the cell or the
particle comb run a multigroup kernel too (csrc/mc_event_kernels.cuh, FL_MGS and FL_MGX:
per-CTA sums in shared memory, so one launch below the history count that
takes replicas): the tile kernel's tallies, and with the comb, which that
kernel has not, FP64 replay's."""
import os
import re

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

N = 100_000


def _write(d, kind):
    from mcgpu import workloads as W
    os.makedirs(d, exist_ok=True)
    W.mg_deep_slab(d, n_regions=4, G=7, thickness=60.0)
    with open(d + "/input.xml") as f:
        s = f.read()
    cells = "".join(f'<cell name="{c}"/>' for c in re.findall(r'<cell name="([^"]+)" material', s))
    if kind == "comb":
        s = s.replace("<population_control>", '<population_control><particle_comb bank_max="4" teeth="3"/>')
        extra = f'<estimator name="x" scores="flux">{cells}<filter type="group"/></estimator>'
    else:
        filt = {"time": '<filter type="time" grid_linear="0.0 2e-9 2e-8"/>',
                "group and time": '<filter type="group"/><filter type="time" grid_linear="0.0 2e-9 2e-8"/>',
                "two": '<filter type="group"/><filter type="energy" grid="-1 1 1e9"/>'}[kind]
        extra = "".join(f'<estimator name="x{t}" type="{t}" scores="flux absorption">{cells}{filt}</estimator>' for t in ("TL", "C"))
    with open(d + "/input.xml", "w") as f:
        f.write(s.replace("</estimators>", extra + "</estimators>"))
    return d


@pytest.mark.parametrize("kind", ["time", "group and time", "two"])
def test_equals_the_tile_kernel(tmp_path, kind):
    import mcgpu
    p = mcgpu.Problem(_write(str(tmp_path), kind))
    out = []
    for kernel in (1, 2):
        p.reset()
        c = p.run(n=N, seed=9, mode="event", kernel=kernel)
        assert c["launches"] == 1
        out.append((*p.all_tallies()[2:], c["tally_updates"], c["xs_evals"], c["flights"]))
    p.close()
    (s1, q1, *c1), (s, q, *c2) = out
    assert c1 == c2 and np.any(s)
    # the same terms in another order: n 2^-53 for a sum of nonnegative ones
    tol = 8 * N * 2.0 ** -53
    assert np.all(np.abs(s - s1) <= tol * s1) and np.all(np.abs(q - q1) <= tol * q1)


def test_comb_agrees_with_replay(tmp_path):
    import mcgpu
    p = mcgpu.Problem(_write(str(tmp_path), "comb"))
    m, sg, s, _ = (a.copy() for a in _run(p, "replay"))
    me, sge, se, _ = _run(p, "event", kernel=2)
    assert p.counters()["launches"] == 1
    p.close()
    seen = (s > 50.0) & (se > 50.0)       # bins with enough histories for a normal bound
    assert np.count_nonzero(seen) >= 8
    z = np.abs(m - me)[seen] / np.sqrt(sg ** 2 + sge ** 2)[seen]
    assert np.all(z < 5.0), z


def _run(p, mode, **kw):
    p.reset()
    p.run(n=N, seed=9, mode=mode, **kw)
    return p.all_tallies()


def test_batch_with_one_time_filter_equals_its_problems(tmp_path):
    import mcgpu
    ds = [_write(str(tmp_path / k.replace(" ", "_")), k) for k in ("two", "time", "two")]
    n = [5000, 20_000, 1]
    ps = [mcgpu.Problem(d) for d in ds]
    b = mcgpu.Batch(ps, n)
    b.reset()
    b.run(seed=4)
    got = b.tallies()[2].copy()
    b.close()
    want = []
    for i, p in enumerate(ps):
        p.reset()
        p.run(n=n[i], seed=mcgpu.batch_problem_seed(4, i), mode="event", kernel=2)
        want.append(p.all_tallies()[2])
        p.close()
    want = np.concatenate(want)
    assert np.any(want) and np.all(np.abs(got - want) <= 8 * max(n) * 2.0 ** -53 * want)
