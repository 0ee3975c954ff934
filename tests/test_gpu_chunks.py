"""FP64 runs in several launches of odd sizes (csrc/mc_engine.cpp, mc_lr.cpp):
columns padded to whole vectors, a short last launch, few lanes a warp.
Replay equals the oracle bit for bit; derivatives over many launches equal the
same histories' of a problem narrow enough for one."""
import numpy as np
import pytest

from helpers import same_bits

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("chunk", [1, 7, 61, 700])
def test_replay_in_odd_chunks_equals_the_oracle(oracle_lib, tmp_path, chunk):
    import mcgpu
    from mcgpu import workloads as W
    d = W.mg_layered_slab(str(tmp_path), n_regions=4, detectors=True)
    n = min(2003, 40 * chunk + 3)
    p = mcgpu.Problem(d)
    p.run(n=n, seed=7, mode="replay", chunk=chunk)
    _, _, s, q = p.all_tallies()
    r = oracle_lib.run(oracle_lib.load(d), n=n, seed=7)
    assert same_bits(s, r.sum) and same_bits(q, r.sq)
    p.reset()
    p.run(n=n, seed=7, mode="plain", chunk=chunk)
    _, _, sp, qp = p.all_tallies()
    p.close()
    # plain mode's own functions and order: a few roundings a flight of some
    # hundred, then n 2^-53 for the sums
    assert np.all(np.abs(sp - s) <= 1e-11 * s) and np.all(np.abs(qp - q) <= 1e-11 * q)


def test_derivatives_over_several_launches(tmp_path):
    import mcgpu
    from mcgpu import workloads as W
    (tmp_path / "a").mkdir()
    (tmp_path / "b").mkdir()
    narrow = W.mg_layered_slab(str(tmp_path / "a"), n_regions=4, detectors=True)
    wide = W.mg_layered_slab(str(tmp_path / "b"), n_regions=4, detectors=True)
    with open(wide + "/input.xml") as f:
        s = f.read()
    pad = '<estimator name="w" scores="flux"><cell name="c0"/><filter type="energy" grid_linear="0 1 20000"/></estimator>'
    with open(wide + "/input.xml", "w") as f:
        f.write(s.replace("</estimators>", pad + "</estimators>"))
    n = 3001                       # launches of some 516 histories
    out = []
    for d in (narrow, wide):
        p = mcgpu.Problem(d)
        par = p.lr_params()
        g, sg = p.backward(par, n, seed=5)
        m, sm = p.forward(par, n, seed=5)
        out.append((g, sg, m, sm))
        p.close()
    k = out[0][0].shape[0]
    assert np.any(out[0][0])
    for a, b in zip(out[0], out[1]):
        assert same_bits(a, b[:k])
