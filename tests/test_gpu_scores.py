"""Tally rows of the per-thread mixed kernel: touched sectors of four bins, in a
register up to 256 bins and in memory beyond (csrc/mc_event_kernels.cuh,
warp_fold), and one attachment record per score, reaction scores with the
flight's cross sections.  The tile kernel runs the same histories with a bit
per bin."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

N = 6000
SCORES = "flux absorption scatter capture total"


def _write(d, kind, regions, general):
    from mcgpu import workloads as W
    if kind == "ce":
        W.slab_1g(d, n_flux_bins=regions, thickness=6.0)
    else:
        W.mg_layered_slab(d, samples=100, n_regions=regions)
    cells = "".join(f'<cell name="c{i}"/>' for i in range(regions))
    two = '<filter type="energy" grid="-1 1e3 1e9"/>' * 2 if general else ""
    extra = "".join(f'<estimator name="x{t}" type="{t}" scores="{SCORES}">{cells}{two}</estimator>' for t in ("TL", "C"))
    with open(d + "/input.xml") as f:
        s = f.read()
    with open(d + "/input.xml", "w") as f:
        f.write(s.replace("</estimators>", extra + "</estimators>"))


# regions: rows of one sector and less, around 256 bins, and of several mask words
@pytest.mark.parametrize("kind,regions", [("ce", 1), ("ce", 21), ("ce", 22), ("ce", 70), ("mg", 1), ("mg", 16), ("mg", 30)])
@pytest.mark.parametrize("general", [False, True])
def test_rows_and_scores(tmp_path, kind, regions, general):
    import mcgpu
    d = str(tmp_path)
    _write(d, kind, regions, general)
    out = []
    for kernel in (1, 2):
        p = mcgpu.Problem(d, d + "/xs_library" if kind == "ce" else None)
        c = p.run(n=N, seed=11, mode="event", kernel=kernel)
        s, q = p.all_tallies()[2:]
        out.append((s.copy(), q.copy(), c["tally_updates"], c["xs_evals"]))
        p.close()
    (s1, q1, t1, x1), (s, q, t2, x2) = out
    assert t1 == t2 and x1 == x2
    # the same terms in another order: n 2^-53 for a sum of nonnegative ones
    tol = 4 * N * 2.0 ** -53
    assert np.all(np.abs(s - s1) <= tol * s1) and np.all(np.abs(q - q1) <= tol * q1)
    filt = 4 if general else 1
    for part in s[-10 * regions * filt:].reshape(2, 5, regions * filt):
        flux, absorption, scatter, capture, total = part
        assert np.count_nonzero(total) >= min(regions, 4)
        assert np.all(np.abs(absorption - capture) <= tol * capture)
        # Sigma_s + Sigma_c = Sigma_t up to one rounding each of the three
        # tables' values and of the three products
        assert np.all(np.abs(scatter + capture - total) <= 6 * 2.0 ** -24 * total)
        assert np.array_equal(flux > 0, total > 0)
