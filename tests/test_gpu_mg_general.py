"""Multigroup problems whose estimators filter twice (no record, no time
filter) run a kernel without the time filters' pair lists
(csrc/mc_event_kernels.cuh, FL_MGS): the second filter, one search in three
values, costs little, and a batch with such problems gives their tallies."""
import os
import re

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

GROUP = '<filter type="group"/>'
TWO = GROUP + '<filter type="energy" grid="-1 1 1e9"/>'


def _problem(folder, filters, regions=8, G=2):
    import mcgpu
    from mcgpu import workloads as W
    d = str(folder)
    os.makedirs(d)
    W.mg_deep_slab(d, n_regions=regions, G=G, thickness=15.0 * regions)
    with open(d + "/input.xml") as f:
        s = f.read()
    cells = "".join(f'<cell name="{c}"/>' for c in re.findall(r'<cell name="([^"]+)" material', s))
    est = "".join(f'<estimator name="x{t}" type="{t}" scores="flux absorption scatter total">{cells}{filters}</estimator>'
                  for t in ("TL", "C"))
    with open(d + "/input.xml", "w") as f:
        f.write(s.replace("</estimators>", est + "</estimators>"))
    return mcgpu.Problem(d)


def test_a_second_filter_costs_little(tmp_path):
    ms = []
    for k, filters in enumerate((GROUP, TWO)):
        p = _problem(tmp_path / str(k), filters)
        t = []
        for r in range(7):
            p.reset()
            t.append(p.run(n=1_000_000, seed=5, mode="event", kernel=2)["total_ms"])
        p.close()
        ms.append(min(t[2:]))
    assert ms[1] <= 1.2 * ms[0], ms


@pytest.mark.parametrize("n", [1, 127, 129, 40_000, (1 << 18) + 1])
def test_equals_the_tile_kernel(tmp_path, n):
    p = _problem(tmp_path / "p", TWO, regions=3, G=7)
    out = []
    for kernel in (1, 2):
        p.reset()
        c = p.run(n=n, seed=9, mode="event", kernel=kernel)
        out.append((*p.all_tallies()[2:], [c[k] for k in ("flights", "collisions", "crossings", "tally_updates", "particles", "splits", "xs_evals")]))
    p.close()
    (s1, q1, c1), (s, q, c2) = out
    assert c1 == c2 and np.any(s)
    # the same terms in another order: n 2^-53 for a sum of nonnegative ones,
    # and some hundred terms in a history
    tol = 8 * (n + 1000) * 2.0 ** -53
    assert np.all(np.abs(s - s1) <= tol * s1) and np.all(np.abs(q - q1) <= tol * q1)


def test_batch_equals_its_problems(tmp_path):
    import mcgpu
    ps = [_problem(tmp_path / str(k), f, r, g) for k, (f, r, g) in enumerate(((TWO, 3, 2), (GROUP, 2, 30), (TWO, 12, 7)))]
    n = [5000, 20_000, 1]
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
    assert np.any(want) and np.all(np.abs(got - want) <= 8 * (max(n) + 1000) * 2.0 ** -53 * want)
