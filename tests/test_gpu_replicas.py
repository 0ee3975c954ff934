"""Long mixed runs fold into replicated sums (csrc/mc_event.cu,
kReplicaHistories): the same tallies as the shared-memory sums of shorter
runs, also after autotuning has folded samples into scratch sums."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("tuned", [False, True])
def test_long_run_equals_the_sum_of_short_ones(tmp_path, tuned):
    import mcgpu
    from mcgpu import workloads as W
    d = W.slab_1g(str(tmp_path), n_flux_bins=70)
    p = mcgpu.Problem(d, d + "/xs_library")
    if tuned:
        p.autotune()
        assert p.histories_run() == 0 and not np.any(p.all_tallies()[2])
    n = 65_536 + 333
    c = p.run(n=n, seed=5, mode="event", kernel=2)
    assert c["launches"] == 2
    _, _, s, q = p.all_tallies()
    p.reset()
    for first in range(0, n, 40_000):
        assert p.run(n=min(40_000, n - first), first=first, seed=5, mode="event", kernel=2)["launches"] == 1
    _, _, s2, q2 = p.all_tallies()
    p.close()
    assert np.count_nonzero(s) > 100
    # the same histories' totals in another order: n 2^-53 bounds the relative
    # difference of two FP64 sums of nonnegative terms
    tol = n * 2.0 ** -53
    assert np.all(np.abs(s - s2) <= 2 * tol * s) and np.all(np.abs(q - q2) <= 2 * tol * q)
