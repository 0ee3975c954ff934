"""Long multigroup runs whose rows fold into replicas keep no wide sums in
shared memory (csrc/mc_event.cu, kWideSums): bins that nothing scores cost a
problem of 3,960 bins what they cost one of 4,140, which has no such sums; and
the tallies on both sides of the line are the same."""
import os
import re

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _problem(folder, bins):
    import mcgpu
    from mcgpu import workloads as W
    d = str(folder)
    os.makedirs(d)
    W.mg_deep_slab(d, n_regions=3, G=30, thickness=45.0)
    with open(d + "/input.xml") as f:
        s = f.read()
    cells = "".join(f'<cell name="{c}"/>' for c in re.findall(r'<cell name="([^"]+)" material', s))
    grid = " ".join("%g" % (1e9 * k) for k in range(1, bins))     # every group's energy is below the second point
    est = f'<estimator name="x" scores="flux">{cells}<filter type="group"/><filter type="energy" grid="-1 1 {grid}"/></estimator>'
    with open(d + "/input.xml", "w") as f:
        f.write(s.replace("</estimators>", est + "</estimators>"))
    return mcgpu.Problem(d)


def _run(p, n, reps=1):
    t = []
    for _ in range(reps):
        p.reset()
        t.append(p.run(n=n, seed=5, mode="event", kernel=2)["total_ms"])
    _, _, s, q = p.all_tallies()
    return min(t), s[s > 0], q[s > 0]


def test_wide_sums_cost_no_shared_memory(tmp_path):
    ms = []
    for bins in (44, 46):
        p = _problem(tmp_path / str(bins), bins)
        ms.append(_run(p, 1_000_000, 7)[0])
        p.close()
    assert ms[0] <= 1.1 * ms[1], ms


@pytest.mark.parametrize("n", [(1 << 18) - 1, (1 << 18) + 1])
def test_same_tallies_at_every_width(tmp_path, n):
    out = []
    for bins in (2, 11, 12, 44, 46):       # around 1,024 bins and 4,096
        p = _problem(tmp_path / str(bins), bins)
        out.append(_run(p, n)[1:])
        p.close()
    # the same histories' totals in another order: n 2^-53 bounds the relative
    # difference of two FP64 sums of nonnegative terms, and histories have
    # some hundred
    tol = 2 * (n + 1000) * 2.0 ** -53
    for s, q in out[1:]:
        assert len(s) == len(out[0][0]) > 0
        assert np.all(np.abs(s - out[0][0]) <= tol * s) and np.all(np.abs(q - out[0][1]) <= tol * q)
