"""Long multigroup runs with estimators on cells fold their history rows into
replicated sums (csrc/mc_event.cu, kReplicaHistoriesMg) and a history's first
bin into shared memory: the same tallies as the sum of shorter runs."""
import re

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

LONG = 1 << 18


# rows of one sector, around a register mask's 256 bins, and currents alone
@pytest.mark.parametrize("regions,groups,flux", [(1, 2, True), (5, 8, True), (8, 30, True), (10, 30, True), (3, 4, False)])
def test_long_multigroup_run_equals_the_sum_of_short_ones(tmp_path, regions, groups, flux):
    import mcgpu
    from mcgpu import workloads as W
    d = W.mg_deep_slab(str(tmp_path), n_regions=regions, G=groups, thickness=20.0 * regions)
    if flux:
        with open(d + "/input.xml") as f:
            s = f.read()
        cells = "".join(f'<cell name="{c}"/>' for c in re.findall(r'<cell name="([^"]+)" material', s))
        est = f'<estimator name="g" scores="flux">{cells}<filter type="group"/></estimator>'
        with open(d + "/input.xml", "w") as f:
            f.write(s.replace("</estimators>", est + "</estimators>"))
    p = mcgpu.Problem(d)
    n = LONG + 333
    for _ in range(2):      # the second run finds the replicas cleared by the first
        p.reset()
        c = p.run(n=n, seed=5, mode="event", kernel=2)
        assert c["launches"] == (2 if flux else 1)
        _, _, s, q = p.all_tallies()
    p.reset()
    for first in range(0, n, 200_000):
        assert p.run(n=min(200_000, n - first), first=first, seed=5, mode="event", kernel=2)["launches"] == 1
    _, _, s2, q2 = p.all_tallies()
    p.close()
    assert np.any(s)
    # the same histories' totals in another order: n 2^-53 bounds the relative
    # difference of two FP64 sums of nonnegative terms
    tol = n * 2.0 ** -53
    assert np.all(np.abs(s - s2) <= 2 * tol * s) and np.all(np.abs(q - q2) <= 2 * tol * q)
