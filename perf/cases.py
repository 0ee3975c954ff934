"""The work that users of this framework have it do, as measurable cases.

A case is one pass of a fixed-source run through the Python entry points
(``Problem``, ``Batch``): tallies cleared, a range of histories run in one of
the three modes, every tally read back; or one forward / backward pair of the
one-group derivative path.  Inputs are the synthetic problems of
``mcgpu.workloads`` and one continuous-energy slab with the population
controls and tally options in use, written to a folder of this process and
read by the library as a user's input is.  The seed picks the Monte Carlo
stream (and the parameter point of a derivative run).

Kinds:
  shield    continuous-energy three-shell sphere: the reference's headline
            kind of problem (deep spectra, free-gas scatter, energy tallies)
  slab      one-group slab cut into many cells, a flux bin in each
  deep      multigroup deep-penetration slab: importance splitting, weight
            roulette, group tallies
  layered   one-group layered slab (also the differentiation problem)
  duct      continuous-energy slab with reflective and vacuum sides, splitting,
            collision and track-length tallies; optional time filter and comb
  batch     many uneven multigroup shields in one launch
Modes: "event" (mixed precision), "plain" and "replay" (FP64; replay is the
interface's default), "forward" / "backward" (FP64 derivatives).
"""
import atexit
import functools
import math
import os
import shutil
import sys
import tempfile

import numpy as np

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
sys.path.insert(0, os.path.join(ROOT, "mc-old_gb300"))

import mcgpu  # noqa: E402
from mcgpu import workloads as W  # noqa: E402


def listed():
    return [
        # a production shielding run: the benchmark problem at its own size
        {"name": "shield event 1e7", "kind": "shield", "mode": "event", "n": 10_000_000, "points": 20_000, "bins": 50},
        # the same problem as a quick look, or one step of an outer loop: too few histories to fill the GPU
        {"name": "shield event 2e4", "kind": "shield", "mode": "event", "n": 20_000, "points": 20_000, "bins": 50},
        # a flux map on a fine mesh of cells, a history crossing many of them
        {"name": "slab event 1e6", "kind": "slab", "mode": "event", "n": 1_000_000, "cells": 100, "thickness": 20.0},
        # deep penetration with variance reduction, the largest history count
        {"name": "deep event 1e8", "kind": "deep", "mode": "event", "n": 100_000_000, "regions": 5, "groups": 30},
        # a small one-group problem, odd history count: launch and read-back latency
        {"name": "layered event 99991", "kind": "layered", "mode": "event", "n": 99_991, "regions": 16},
        # a parameter scan: uneven shields together in one launch
        {"name": "batch event 256", "kind": "batch", "mode": "event", "problems": 256, "least": 1000, "most": 1_000_000},
        # the verified FP64 run a user starts with (the interface's default mode)
        {"name": "shield replay 5e4", "kind": "shield", "mode": "replay", "n": 50_000, "points": 20_000, "bins": 50},
        # every population control and tally option at once, a few thousand histories: the smallest call
        {"name": "duct replay 3001", "kind": "duct", "mode": "replay", "n": 3001, "points": 400, "time": True, "comb": 0},
        # FP64 without the replay's portable functions: the double-precision check of a mixed run
        {"name": "shield plain 2e5", "kind": "shield", "mode": "plain", "n": 200_000, "points": 20_000, "bins": 50},
        {"name": "deep plain 2e6", "kind": "deep", "mode": "plain", "n": 2_000_000, "regions": 5, "groups": 30},
        # a bitwise reproducible run of a multigroup problem
        {"name": "layered replay 5e5", "kind": "layered", "mode": "replay", "n": 500_000, "regions": 16},
        # gradients of all currents with respect to every layer's cross sections
        {"name": "layered backward 5e4", "kind": "layered", "mode": "backward", "n": 50_000, "regions": 16},
    ]


# histories of drawn cases: (least, most) for each kind and mode
RANGES = {
    ("shield", "event"): (1e4, 1e7), ("slab", "event"): (1e4, 4e6), ("deep", "event"): (1e5, 1e8),
    ("layered", "event"): (1e4, 2e7), ("duct", "event"): (1e4, 5e5),
    ("shield", "plain"): (2e3, 2e5), ("slab", "plain"): (5e3, 5e5), ("deep", "plain"): (1e4, 2e6),
    ("layered", "plain"): (1e4, 2e6), ("duct", "plain"): (2e3, 3e4),
    ("shield", "replay"): (1e3, 5e4), ("slab", "replay"): (2e3, 1e5), ("deep", "replay"): (5e3, 3e5),
    ("layered", "replay"): (5e3, 5e5), ("duct", "replay"): (1e3, 1e4),
    ("layered", "forward"): (5e3, 3e5), ("layered", "backward"): (2e3, 5e4),
    ("batch", "event"): (8, 256),
}


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind, mode = rng.choice(sorted(RANGES))
    n = _log_int(rng, *RANGES[kind, mode])
    if kind == "shield":
        return {"kind": kind, "mode": mode, "n": n, "points": _log_int(rng, 300, 20_000), "bins": rng.randint(3, 150)}
    if kind == "slab":
        return {"kind": kind, "mode": mode, "n": n, "cells": _log_int(rng, 10, 150), "thickness": rng.uniform(5.0, 20.0)}
    if kind == "deep":
        return {"kind": kind, "mode": mode, "n": n, "regions": rng.randint(2, 6), "groups": rng.randint(2, 30)}
    if kind == "layered":
        return {"kind": kind, "mode": mode, "n": n, "regions": rng.randint(2, 16)}
    if kind == "duct":
        return {"kind": kind, "mode": mode, "n": n, "points": _log_int(rng, 50, 2000), "time": rng.random() < 0.5,
                "comb": rng.choice((0, 0, 2, 5))}
    return {"kind": kind, "mode": mode, "problems": n, "least": 1000, "most": _log_int(rng, 1e5, 1e6)}


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------
@functools.lru_cache(maxsize=None)
def _folder():
    d = tempfile.mkdtemp(prefix="mcgpu_cases_")
    atexit.register(shutil.rmtree, d, ignore_errors=True)
    return d


_DUCT_CELLS = (("water", 1.0), ("carbon", 3.0), ("water", 9.0), (None, 4.0), ("carbon", 2.0))


def _duct(d, points, time, comb):
    """2 cm layers between reflective y and vacuum z sides, split by importance."""
    os.makedirs(os.path.join(d, "xs_library"))
    E = np.exp(np.linspace(math.log(1e-5), math.log(2e7), points))
    for zaid, A, s0, Ec, c0 in (("700001", 1.0, 6.0, 1e6, 0.3), ("700016", 16.0, 4.0, 3e6, 0.05),
                                ("700012", 12.0, 5.0, 2e6, 0.01)):
        W.write_xs_table(os.path.join(d, "xs_library", zaid + ".txt"), A, E, s0 / (1.0 + E / Ec), c0 * np.sqrt(0.0253 / E))
    names = ["r%d" % i for i in range(len(_DUCT_CELLS))]
    solid = [c for c, (m, _) in zip(names, _DUCT_CELLS) if m]
    x = ["<?xml version = '1.0' encoding = 'UTF-8'?>\n<simulation>\n    <description name=\"duct\" samples=\"1000\"/>\n</simulation>\n"]
    if comb:
        x.append('<population_control>\n    <particle_comb bank_max="%d" teeth="%d"/>\n</population_control>\n' % (comb + 1, comb))
    x.append('<nuclides>\n    <nuclide name="H" ZAID="700001"/>\n    <nuclide name="O" ZAID="700016"/>\n    <nuclide name="C" ZAID="700012"/>\n</nuclides>\n')
    x.append('<materials>\n    <material name="water"><nuclide name="H" density="0.06"/><nuclide name="O" density="0.03"/></material>\n'
             '    <material name="carbon"><nuclide name="C" density="0.09"/></material>\n</materials>\n<surfaces>\n')
    x += ['    <plane_x name="x%d" x="%g"/>\n' % (i, 2.0 * i) for i in range(len(names) + 1)]
    x.append('    <plane_y name="ylo" y="-3.0" bc="reflective"/>\n    <plane_y name="yhi" y="3.0" bc="reflective"/>\n'
             '    <plane_z name="zlo" z="-4.0" bc="vacuum"/>\n    <plane_z name="zhi" z="4.0" bc="vacuum"/>\n</surfaces>\n<cells>\n')
    for i, (m, imp) in enumerate(_DUCT_CELLS):
        x.append('    <cell name="r%d"%s importance="%g">\n        <surface name="x%d" sense="+1"/><surface name="x%d" sense="-1"/>\n'
                 '        <surface name="ylo" sense="+1"/><surface name="yhi" sense="-1"/>\n'
                 '        <surface name="zlo" sense="+1"/><surface name="zhi" sense="-1"/>\n    </cell>\n'
                 % (i, ' material="%s"' % m if m else "", imp, i, i + 1))
    x.append('    <cell name="left" importance="0.0"><surface name="x0" sense="-1"/></cell>\n'
             '    <cell name="right" importance="0.0"><surface name="x%d" sense="+1"/></cell>\n</cells>\n' % len(names))
    x.append('<distributions>\n    <uniform name="Eu" datatype="double" a="1e5" b="2e6"/>\n    <uniform name="ux" datatype="double" a="0.3" b="1.0"/>\n'
             '    <uniform name="uy" datatype="double" a="-0.4" b="0.4"/>\n    <delta name="uz" datatype="double" val="0.1"/>\n'
             '    <independentXYZ name="beam" datatype="point" x="ux" y="uy" z="uz"/>\n    <isotropic name="iso" datatype="point"/>\n'
             '    <delta name="E1" datatype="double" val="1.5e6"/>\n</distributions>\n<sources>\n'
             '    <point x="1e-6" y="0.5" z="-0.25" direction="beam" energy="Eu"/>\n    <point x="1.0" y="0.0" z="0.0" direction="iso" energy="E1"/>\n</sources>\n')
    cells = lambda which: "".join('<cell name="%s"/>' % c for c in which)  # noqa: E731
    x.append('<estimators>\n    <estimator name="tl" scores="flux absorption scatter">\n        %s\n'
             '        <filter type="energy" grid_lethargy="1e-5 2e7 10"/>\n    </estimator>\n' % cells(solid))
    x.append('    <estimator name="coll" type="C" scores="absorption total">\n        %s\n    </estimator>\n' % cells(solid))
    x.append('    <estimator name="out" scores="cross">\n        <surface name="x0"/><surface name="x%d"/>\n    </estimator>\n' % len(names))
    if time:
        x.append('    <estimator name="when" scores="flux">\n        %s\n        <filter type="time" grid_linear="0.0 2e-9 2e-8"/>\n'
                 '    </estimator>\n' % cells(names))
    x.append("</estimators>\n")
    with open(os.path.join(d, "input.xml"), "w") as f:
        f.write("".join(x))


@functools.lru_cache(maxsize=None)
def _written(kind, *size):
    """Writes the input of one problem (or of a batch) once per process: its folder, or [(folder, histories), ...]."""
    d = tempfile.mkdtemp(dir=_folder())
    if kind == "shield":
        W.ce_sphere(d, n_points=size[0], n_spectrum=size[1])
    elif kind == "slab":
        W.slab_1g(d, n_flux_bins=size[0], thickness=size[1])
    elif kind == "deep":
        W.mg_deep_slab(d, n_regions=size[0], G=size[1], thickness=20.0 * size[0])
    elif kind == "layered":
        W.mg_layered_slab(d, n_regions=size[0], detectors=True)
    elif kind == "duct":
        _duct(d, *size)
    else:
        return W.batch_shields(d, n_problems=size[0], min_hist=size[1], max_hist=size[2])
    return d


SIZE_KEYS = {"shield": ("points", "bins"), "slab": ("cells", "thickness"), "deep": ("regions", "groups"),
             "layered": ("regions",), "duct": ("points", "time", "comb"), "batch": ("problems", "least", "most")}


def _load(d):
    xs = os.path.join(d, "xs_library")
    return mcgpu.Problem(d, xs if os.path.isdir(xs) else None)


def _params(p, seed):
    """A parameter point of an outer optimisation: every cross section within 2 % of the input's."""
    own = p.lr_params()
    return own * np.random.default_rng(seed).uniform(0.98, 1.02, own.size)


def prepare(case, seed):
    where = _written(case["kind"], *(case[k] for k in SIZE_KEYS[case["kind"]]))
    s = {"mode": case["mode"], "seed": 1 + seed, "n": case.get("n")}
    if case["kind"] == "batch":
        s["batch"] = mcgpu.Batch([_load(d) for d, _ in where], [n for _, n in where])
    else:
        s["problem"] = _load(where)
        if case["mode"] in ("forward", "backward"):
            s["params"] = _params(s["problem"], seed)
    return s


COUNTS = ("flights", "collisions", "crossings", "tally_updates", "particles", "splits", "xs_evals", "freegas_iters",
          "nuc_lookups", "histories")


def _answer(tallies, counters):
    return dict(zip(("mean", "sigma", "sum", "sumsq"), tallies),
                counts=np.array([counters[k] for k in COUNTS], np.int64))


def run(state):
    p = state.get("problem")
    if state["mode"] == "forward":
        return dict(zip(("mean", "sigma"), p.forward(state["params"], state["n"], seed=state["seed"])))
    if state["mode"] == "backward":
        return dict(zip(("gradient", "sigma"), p.backward(state["params"], state["n"], seed=state["seed"])))
    if p is None:
        b = state["batch"]
        b.reset()
        c = b.run(seed=state["seed"])
        return _answer(b.tallies(), c)
    p.reset()
    c = p.run(n=state["n"], seed=state["seed"], mode=state["mode"])
    return _answer(p.all_tallies(), c)


# ---------------------------------------------------------------------------
# what a pass cannot do without
# ---------------------------------------------------------------------------
# events of one history (flights) of each kind at its listed size, and the
# arithmetic of one event: the exponential and distance of a flight, the
# nearest surface, cross sections, the outgoing direction or velocity, tallies
EVENTS = {"shield": 115.0, "slab": 18.0, "deep": 5.0, "layered": 6.0, "duct": 60.0, "batch": 9.0}
EVENT_FLOPS = {"shield": 300.0, "slab": 90.0, "deep": 80.0, "layered": 80.0, "duct": 250.0, "batch": 90.0}


def work(case):
    kind = case["kind"]
    bins = {"shield": lambda: 4 + case["bins"], "slab": lambda: 2 + 2 * case["cells"],
            "deep": lambda: 1 + case["groups"], "layered": lambda: 3 + case["regions"],
            "duct": lambda: 180 if case["time"] else 130, "batch": lambda: 5 * case["problems"]}[kind]()
    tables = {"shield": lambda: 5 * 4 * 8 * case["points"], "slab": lambda: 300 * case["cells"],
              "deep": lambda: 8 * case["regions"] * (2 + case["groups"]) * case["groups"],
              "layered": lambda: 300 * case["regions"], "duct": lambda: 3 * 4 * 8 * case["points"],
              "batch": lambda: 3000 * case["problems"]}[kind]()
    if kind == "batch":
        n = case["problems"] * (case["most"] - case["least"]) / math.log(case["most"] / case["least"])
    else:
        n = case["n"]
    flops = n * EVENTS[kind] * EVENT_FLOPS[kind]
    columns = 1
    if case["mode"] == "backward":   # the score function's two numbers a flight; every crossing scores all derivatives
        columns = 2 * case["regions"]
        flops += n * EVENTS[kind] * 3 * columns
    return {"bytes": tables + 4 * 8 * bins * columns, "flops": flops}


# ---------------------------------------------------------------------------
# 64-bit values where plain numpy can follow the histories
# ---------------------------------------------------------------------------
def _philox(b, event, ident, hist, key):
    c = [np.full(hist.shape, b, np.uint64), event.astype(np.uint64), ident, (hist & 0xFFFFFFFF).astype(np.uint64)]
    k0, k1 = key
    low = np.uint64(0xFFFFFFFF)
    for r in range(10):
        p0, p1 = c[0] * np.uint64(0xD2511F53), c[2] * np.uint64(0xCD9E8D57)
        c = [(p1 >> np.uint64(32)) ^ c[1] ^ np.uint64(k0), p1 & low, (p0 >> np.uint64(32)) ^ c[3] ^ np.uint64(k1), p0 & low]
        k0, k1 = (k0 + 0x9E3779B9) & 0xFFFFFFFF, (k1 + 0xBB67AE85) & 0xFFFFFFFF
    return c


def _uniforms(event, hist, key, draws):
    """The first draws of one event of each history's only particle, as 64-bit uniforms in (0, 1)."""
    out = []
    for b in range((draws + 1) // 2):
        w = _philox(b, event, np.zeros(hist.shape, np.uint64), hist, key)
        for lo, hi in ((w[0], w[1]), (w[2], w[3])):
            v = ((hi << np.uint64(32)) | lo) >> np.uint64(12)
            out.append((v.astype(np.float64) + 0.5) * 2.0 ** -52)
    return out[:draws]


def _follow(scat, absb, n, seed, derivatives):
    """Histories of the layered one-group slab (1 cm layers, detectors on every plane) as arrays: per-history bin
    totals, and with derivatives their products with the score function of every (Sigma_s, Sigma_a)."""
    R = scat.size
    tot = scat + absb
    cap = tot - scat
    K = 2 * R
    hist = np.arange(n, dtype=np.uint64)
    key = (seed & 0xFFFFFFFF, seed >> 32)
    bins = 2 + R + 1
    rows = np.zeros((n, bins))
    drows = np.zeros((n, bins, K)) if derivatives else None
    S = np.zeros((n, K)) if derivatives else None
    u = _uniforms(np.zeros(n, np.uint64), hist, key, 3)
    mu, azi = u[1], 2.0 * np.pi * u[2]
    c = np.sqrt(1.0 - mu * mu)
    d = np.stack([mu, np.cos(azi) * c, np.sin(azi) * c])
    x, w, cell = np.full(n, 1e-9), np.ones(n), np.zeros(n, np.int64)
    at = np.arange(n)          # the history of each particle still walking
    eps, far = float(np.finfo(np.float32).eps), float(np.finfo(np.float32).max)
    event = 0
    while at.size:
        event += 1
        u = _uniforms(np.full(at.size, event, np.uint64), hist[at], key, 5)
        with np.errstate(divide="ignore"):
            dl = np.where(np.abs(d[0]) > eps, (cell - x) / d[0], far)
            dr = np.where(np.abs(d[0]) > eps, (cell + 1.0 - x) / d[0], far)
        dl, dr = np.where(dl > 0.0, dl, far), np.where(dr > 0.0, dr, far)
        plane = np.where(dl <= dr, cell, cell + 1)
        dist = np.minimum(dl, dr)
        dcol = -np.log(u[0]) / tot[cell]
        crosses = dcol > dist
        step = np.where(crosses, dist, dcol)
        x = x + d[0] * step
        if derivatives:
            S[at, 2 * cell] -= step
            S[at, 2 * cell + 1] -= step
        alive = np.ones(at.size, bool)
        # crossings: the plane's current, then the next layer or the outside
        i = np.flatnonzero(crosses)
        x[i] = x[i] + d[0, i] * eps
        for b, sel in ((2 + plane[i], np.ones(i.size, bool)), (np.zeros(i.size, np.int64), plane[i] == R),
                       (np.ones(i.size, np.int64), plane[i] == 0)):
            rows[at[i[sel]], b[sel]] += w[i[sel]]
            if derivatives:
                drows[at[i[sel]], b[sel]] += w[i[sel], None] * S[at[i[sel]]]
        cell[i] = np.floor(np.where(x[i] < plane[i], plane[i] - 1, plane[i]))
        alive[i] = (cell[i] >= 0) & (cell[i] < R)
        # collisions: implicit capture, then an isotropic direction
        j = np.flatnonzero(~crosses)
        m = cell[j]
        if derivatives:
            S[at[j], 2 * m] += 1.0 / scat[m]
        w[j] = w[j] * (tot[m] - cap[m]) / tot[m]
        mu, azi = 2.0 * u[2][j] - 1.0, 2.0 * np.pi * u[3][j]
        ca, sa, A = np.cos(azi), np.sin(azi), np.sqrt(1.0 - mu * mu)
        dx, dy, dz = d[:, j]
        B = np.sqrt(1.0 - dz * dz)
        C = A / B
        d[:, j] = (dx * mu + (dx * dz * ca - dy * sa) * C, dy * mu + (dy * dz * ca + dx * sa) * C, dz * mu - ca * A * B)
        # weight roulette (default 0.001 -> 1) with the event's next draw
        low = alive & (w < 0.001)
        last = np.where(crosses, u[1], u[4])
        win = low & (last < w)
        w[win] = 1.0
        alive &= ~(low & ~win)
        at, x, w, cell, d = at[alive], x[alive], w[alive], cell[alive], d[:, alive]
    return rows, drows


def exact(case, seed):
    # the mixed mode's histories are drawn and followed in FP32, and the other problems' histories branch into more
    # particles or take tabulated collisions: no value of a 64-bit restatement here belongs to them
    if case["kind"] != "layered" or case["mode"] == "event":
        return None
    p = _load(_written("layered", case["regions"]))
    n, R = case["n"], case["regions"]
    par = p.lr_params() if case["mode"] in ("plain", "replay") else _params(p, seed)
    p.close()
    rows, drows = _follow(par[0::2], par[1::2], n, 1 + seed, case["mode"] == "backward")

    def mean_sigma(v):
        s, q = v.sum(axis=0), (v * v).sum(axis=0)
        m = s / n
        return m, np.sqrt(np.maximum(0.0, (q / n - m * m) / (n - 1.0))), s, q

    if case["mode"] == "backward":
        m, sg, _, _ = mean_sigma(drows.reshape(n, -1))
        return {"gradient": m.reshape(R + 3, 2 * R), "sigma": sg.reshape(R + 3, 2 * R)}
    m, sg, s, q = mean_sigma(rows)
    if case["mode"] == "forward":
        return {"mean": m, "sigma": sg}
    return {"mean": m, "sigma": sg, "sum": s, "sumsq": q, "counts": None}
