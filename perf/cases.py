"""The calls that programs built on this package make, as timed cases.

Each case is one call of the public interface (``solve``, ``MeshSystem.sweep``,
``batch_sweep``, ``MeshSystem.gradient``, ``MeshSystem.currents``,
``partial_inductance_matrix``, ``IterativeSystem.impedance``) on a synthetic
deck of :mod:`fasterhenry_b200.fixtures`.  A case names its deck by sizes; the
seed varies the lengths (pitch, trace width, thickness, side) by a few per
cent, so two seeds are two layouts of the same size.

* ``listed()``  the cases that are timed by name.
* ``draw(rng)`` one more case from the same ranges.
* ``prepare(case, seed)`` what a program holds before the call: the geometry,
  or the assembled system.
* ``run(state)`` the call, and all the numbers it returns.
* ``work(case)`` the bytes and operations the call cannot do without.
* ``exact(case, seed)`` the same numbers from plain numpy / torch in 64 bits,
  for the decks small enough for it: every filament pair integrated on its
  own, and a nodal (not mesh) solve of the circuit.
"""
import math
import random

import numpy as np
import torch

import fasterhenry_b200 as fh
from fasterhenry_b200 import fixtures as F

UM = 1e-6
MU0 = 4.0e-7 * math.pi
#: Largest system that exact() integrates pair by pair.
EXACT_FILAMENTS = 2500


# ---------------------------------------------------------------------------
# The cases
# ---------------------------------------------------------------------------
def listed():
    return [
        # The smallest whole call: a 4-turn on-chip spiral from geometry to Z
        # at ten frequencies, in the default (FP64) form.  Latency: meshing,
        # a 29k-pair fill and ten factorizations of order 224.
        {"name": "solve_spiral_240", "kind": "solve", "shape": "spiral", "turns": 4, "nw": 5, "nh": 3, "ports": 1,
         "nf": 10, "precision": "fp64"},
        # The large whole call: geometry to Z of a 10,020-filament meander,
        # 32 frequencies, mixed form (fill, congruence and sweep together).
        {"name": "solve_meander_10020", "kind": "solve", "shape": "meander", "legs": 167, "nw": 10, "nh": 3,
         "ports": 1, "nf": 32, "precision": "mixed"},
        # An ordinary sweep in the default FP64 form, two ports.
        {"name": "sweep_2400_fp64", "kind": "sweep", "shape": "meander", "legs": 40, "nw": 10, "nh": 3, "ports": 2,
         "nf": 32, "precision": "fp64"},
        # The same deck in the mixed form, one port.
        {"name": "sweep_2400_mixed", "kind": "sweep", "shape": "meander", "legs": 40, "nw": 10, "nh": 3, "ports": 1,
         "nf": 32, "precision": "mixed"},
        # The large sweep in the mixed form: 9,686 loops, 32 frequencies.
        {"name": "sweep_10020_mixed", "kind": "sweep", "shape": "meander", "legs": 167, "nw": 10, "nh": 3,
         "ports": 1, "nf": 32, "precision": "mixed"},
        # A few frequencies of a large deck of odd order in the FP64 form
        # (29 x 1 per segment, one segment at 30 x 1: 6,553 loops).
        {"name": "sweep_6787_fp64", "kind": "sweep", "shape": "meander", "legs": 117, "nw": 29, "nh": 1,
         "ports": 1, "nf": 5, "precision": "fp64", "ragged": True},
        # A library of 64 uneven spirals at once, 16 frequencies each, mixed.
        {"name": "batch_64_spirals", "kind": "batch", "count": 64, "nf": 16, "precision": "mixed"},
        # One step of an inductor optimization: dZ/dp of every width,
        # thickness and node coordinate of a graded spiral at 1 GHz.
        {"name": "gradient_spiral", "kind": "gradient", "turns": 6, "skin_depths": 0.1, "coordinates": True},
        # Filament currents of a graded 5-turn spiral over a few frequencies.
        {"name": "currents_spiral_900", "kind": "currents", "turns": 5, "nw": 9, "nh": 5, "ratio": 1.5, "nf": 4},
        # The partial-inductance matrix of bars in general position
        # (sampled filaments), to the host.
        {"name": "inductance_cloud_1500", "kind": "inductance", "n": 1500, "manhattan": False},
        # Above the dense path's size the solver choice "auto" goes
        # matrix-free: a whole call with the default parameters.
        {"name": "solve_auto_10200", "kind": "auto", "bars": 50, "nf": 1},
        # Z of the large matrix-free system at one frequency: a square
        # meander of 157 runs over a meshed ground plane (107k filaments),
        # 3 x 3 x 3 stencils, FP32 convolution, GMRES to 1e-8.
        {"name": "matrix_free_107144", "kind": "matrix_free", "bars": 157, "cells": 64, "restart": 400},
    ]


def _log(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def draw(rng):
    kind = rng.choice(["solve", "solve", "sweep", "sweep", "sweep", "batch", "gradient", "currents", "inductance",
                       "auto", "matrix_free"])
    c = {"kind": kind}
    if kind in ("solve", "sweep"):
        precision = rng.choice(["fp64", "mixed"])
        if kind == "solve" and rng.random() < 0.5:
            c.update(shape="spiral", turns=rng.randint(2, 8), nw=rng.randint(3, 10), nh=rng.randint(1, 3))
        else:
            # an FP64 sweep of the large sizes takes seconds: fewer legs
            top = 120 if precision == "fp64" else 167
            c.update(shape="meander", legs=int(_log(rng, 8, top)), nw=rng.randint(4, 10), nh=rng.randint(1, 3))
        c["ragged"] = rng.random() < 0.3
        m = _filaments(c)
        room = 1.2e12 if precision == "fp64" else 2.5e13
        c.update(ports=rng.choice([1, 1, 2, 4]), nf=max(1, min(rng.randint(1, 32), int(room / m ** 3))),
                 precision=precision)
    elif kind == "batch":
        c.update(count=int(_log(rng, 4, 64)), nf=rng.randint(2, 16), precision="mixed")
    elif kind == "gradient":
        c.update(turns=rng.randint(2, 6), skin_depths=rng.uniform(0.1, 0.5), coordinates=rng.random() < 0.7)
    elif kind == "currents":
        c.update(turns=rng.randint(2, 6), nw=rng.randint(3, 13), nh=rng.randint(2, 6), ratio=rng.uniform(1.1, 2.0),
                 nf=rng.randint(1, 6))
    elif kind == "inductance":
        c.update(n=int(_log(rng, 100, 1500)), manhattan=rng.random() < 0.5)
    elif kind == "auto":
        c.update(bars=rng.randint(50, 60), nf=1)
    else:
        bars = int(_log(rng, 50, 150))
        c.update(bars=bars, cells=rng.randint(16, 60), restart=rng.choice([200, 400]))
    return c


# ---------------------------------------------------------------------------
# Decks
# ---------------------------------------------------------------------------
def _filaments(case):
    per = case["nw"] * case["nh"]
    segments = 4 * case["turns"] if case.get("shape", "spiral") == "spiral" else 2 * case["legs"]
    return segments * per + (case["nh"] if case.get("ragged") else 0)


def _tapped(deck, ports):
    """`ports` ports along a chain: port k between the chain's k-th and
    (k+1)-th tap (taps evenly spaced from end to end)."""
    last = len(deck.nodes) - 1
    taps = [round(last * k / ports) for k in range(ports + 1)]
    deck.ports = [(taps[k], taps[k + 1]) for k in range(ports)]
    return deck


def _deck(case, seed):
    r = random.Random(1000003 * int(seed) + 17)

    def near(v, by=0.04):
        return v * r.uniform(1.0 - by, 1.0 + by)

    kind = case["kind"]
    if kind in ("solve", "sweep"):
        disc = F.uniform(case["nw"], case["nh"])
        if case.get("ragged"):
            # one segment with a wider grid than the others
            segments = 4 * case["turns"] if case["shape"] == "spiral" else 2 * case["legs"]
            disc = F.per_segment([(case["nw"] + (k == 5), case["nh"]) for k in range(segments)])
        if case["shape"] == "spiral":
            # room for up to 8 turns at this pitch
            deck = F.square_spiral(case["turns"], near(10 * UM), near(5 * UM), near(2 * UM),
                                   near(max(300, 45 * case["turns"]) * UM), disc)
        else:
            deck = F.meander(case["legs"], near(1e-3), near(40 * UM), near(20 * UM), near(5 * UM), disc)
        return _tapped(deck, case["ports"])
    if kind == "gradient":
        # the width and thickness set the grading's cell counts: fixed
        return F.square_spiral(case["turns"], 15 * UM, near(5 * UM), 3 * UM, near(500 * UM),
                               F.skin_depth(1e9, case["skin_depths"], 1.4))
    if kind == "currents":
        return F.square_spiral(case["turns"], near(12 * UM), near(5 * UM), near(3 * UM), near(400 * UM),
                               F.graded(case["nw"], case["nh"], case["ratio"]))
    if kind == "auto":
        return F.scaling_meander(case["bars"], near(100 * UM), near(20 * UM), near(10 * UM))
    deck = F.meander_over_plane(case["bars"], cells=case["cells"])
    # the meander's traces and the gap below them, by the seed
    width, drop = near(20 * UM), near(50 * UM, 0.1) - 50 * UM
    meander_nodes = {sg["a"] for sg in deck.segments[-case["bars"] * (case["bars"] + 1):]}
    meander_nodes |= {sg["b"] for sg in deck.segments[-case["bars"] * (case["bars"] + 1):]}
    for sg in deck.segments[-case["bars"] * (case["bars"] + 1):]:
        sg["width"] = width
    deck.nodes = [(x, y, z + drop if k in meander_nodes else z) for k, (x, y, z) in enumerate(deck.nodes)]
    return deck


def _batch_decks(case, seed):
    return F.random_spirals(case["count"], seed=2026 + 7919 * int(seed))


def _frequencies(case):
    kind = case["kind"]
    if kind == "solve" and case["shape"] == "spiral":
        return F.logspace(6, 10, case["nf"])
    if kind == "batch":
        return F.logspace(7, 10, case["nf"])
    if kind == "currents":
        return F.logspace(8, 10, case["nf"])
    if kind == "auto":
        return F.logspace(9, 10, case["nf"])
    return F.logspace(5, 10, case["nf"])


_PRECISION = {"fp64": fh.Precision.FP64, "mixed": fh.Precision.MIXED_BF16X3}


# ---------------------------------------------------------------------------
# prepare and run
# ---------------------------------------------------------------------------
def prepare(case, seed):
    kind = case["kind"]
    state = {"kind": kind}
    if kind == "inductance":
        deck = F.cloud_deck(case["n"], case["manhattan"], 4242 + int(seed))
        state["filaments"], _ = fh.discretize(fh.Geometry.from_deck(deck), deck.discretization)
        return state
    state["frequencies"] = _frequencies(case) if kind not in ("gradient", "matrix_free") else [1e9]
    state["precision"] = _PRECISION[case.get("precision", "fp64")]
    if kind == "batch":
        decks = _batch_decks(case, seed)
        state["systems"] = [fh.MeshSystem.assemble(fh.Geometry.from_deck(d), d.ports, d.discretization)
                            for d in decks]
        state["frequencies"] = [state["frequencies"]] * len(decks)
        return state
    deck = _deck(case, seed)
    geometry = fh.Geometry.from_deck(deck)
    if kind in ("solve", "auto"):
        state.update(geometry=geometry, ports=deck.ports, discretization=deck.discretization,
                     solver=fh.SolverChoice.AUTO if kind == "auto" else fh.SolverChoice.DENSE)
    elif kind == "matrix_free":
        params = fh.IterativeParams(
            pfft=fh.PfftParams(near_field_radius=8.0, interpolation_order=2, fft_fp32=True),
            gmres=fh.GmresParams(tolerance=1e-8, restart=case["restart"]))
        state["system"] = fh.IterativeSystem.assemble(geometry, deck.ports, deck.discretization, params)
    else:
        state["system"] = fh.MeshSystem.assemble(geometry, deck.ports, deck.discretization)
    if kind == "gradient":
        segments, nodes = range(len(deck.segments)), range(len(deck.nodes))
        state["params"] = [fh.Param(k, s) for k in ("width", "thickness") for s in segments]
        if case["coordinates"]:
            state["params"] += [fh.Param(k, v) for k in ("x", "y") for v in nodes]
    return state


def run(state):
    kind, freqs = state["kind"], state.get("frequencies")
    if kind in ("solve", "auto"):
        return fh.solve(state["geometry"], state["ports"], state["discretization"], freqs, state["precision"],
                        state["solver"]).impedance_ohm
    if kind == "sweep":
        return state["system"].sweep(freqs, state["precision"]).impedance_ohm
    if kind == "batch":
        return [r.impedance_ohm for r in fh.batch_sweep(state["systems"], freqs, state["precision"])]
    if kind == "gradient":
        g = state["system"].gradient(freqs[0], state["params"])
        return {"impedance": g.impedance_ohm, "gradient": g.gradient}
    if kind == "currents":
        # the filament of largest |J| stays out: the top and the bottom row
        # of a planar spiral carry the same current, so it is a tie
        return [{"current": s.current, "density": s.current_density, "power": s.power_w,
                 "segment_current": s.segment_current, "segment_power": s.segment_power_w,
                 "peak_density": s.peak_current_density} for s in state["system"].currents(freqs)]
    if kind == "inductance":
        return fh.partial_inductance_matrix(state["filaments"])
    return state["system"].impedance(freqs[0])


# ---------------------------------------------------------------------------
# Work
# ---------------------------------------------------------------------------
#: Operations of one pair's mutual inductance by a 2 x 2 x 2 point rule
#: (64 distances), the cheapest rule that the fill takes.
PAIR_FLOPS = 64 * 12.0


def _symmetric_solve(m, p, nf):
    """L D L^T of a complex symmetric matrix of order m, nf times (8 real
    operations per complex multiply-add, m^3 / 6 of them), and 2 m^2 p for
    the solves."""
    return nf * (8.0 * m ** 3 / 6.0 + 8.0 * m * m * p)


def work(case):
    kind = case["kind"]
    if kind in ("solve", "sweep", "currents"):
        n = _filaments(case)
        segments = n // (case["nw"] * case["nh"])
        m, p, nf = n - segments, case.get("ports", 1), case["nf"]
        flops = _symmetric_solve(m, p, nf)
        # each L_m entry of the lower triangle once (a sweep), or the
        # geometry in (a whole call)
        nbytes = 16.0 * nf * p * p + (256.0 * n if kind == "solve" else 4.0 * m * m)
        if kind == "solve":
            flops += PAIR_FLOPS * n * n / 4.0
        if kind == "currents":
            nbytes += nf * n * 32.0
        return {"bytes": nbytes, "flops": flops}
    if kind == "batch":
        flops = nbytes = 0.0
        for d in F.random_spirals(case["count"]):
            per = d.discretization["nw"] * d.discretization["nh"]
            m = len(d.segments) * (per - 1)
            flops += _symmetric_solve(m, 1, case["nf"])
            nbytes += 4.0 * m * m + 16.0 * case["nf"]
        return {"bytes": nbytes, "flops": flops}
    if kind == "gradient":
        delta = 1.0 / math.sqrt(math.pi * 1e9 * MU0 * F.COPPER)
        n = 4 * case["turns"] * _graded_count(15 * UM, delta * case["skin_depths"]) * _graded_count(
            3 * UM, delta * case["skin_depths"])
        rates = 4 + (8 if case["coordinates"] else 0)
        return {"bytes": 8.0 * n * n, "flops": _symmetric_solve(n, 1, 1) + rates * PAIR_FLOPS * n * n / 2.0}
    if kind == "inductance":
        n = case["n"]
        return {"bytes": 152.0 * n + 8.0 * n * n, "flops": PAIR_FLOPS * n * n / 2.0}
    # matrix-free: one product per GMRES step; a step streams the near field
    # (about 600 partners a filament at 12 bytes, half of them by symmetry)
    # and the filaments' vectors.  The fewest steps: 50.
    n = 4 * case["bars"] * (case["bars"] + 1) + 2 * case.get("cells", 0) ** 2
    return {"bytes": 50.0 * (300 * 12.0 + 64.0) * n, "flops": 50.0 * 2.0 * 600 * n}


def _graded_count(extent, target, ratio=1.4, most=32):
    for n in range(1, most + 1):
        if extent / sum(ratio ** min(i, n - 1 - i) for i in range(n)) <= target:
            return n
    return most


# ---------------------------------------------------------------------------
# exact: pair integrals and a nodal solve in plain numpy / torch
# ---------------------------------------------------------------------------
def _cells(extent, n, ratio):
    w = np.array([ratio ** min(i, n - 1 - i) for i in range(n)])
    size = extent * w / w.sum()
    return np.cumsum(size) - 0.5 * size - 0.5 * extent, size


def _bars(deck):
    """The deck's filaments (all in a plane z = const, along x or y): axis
    (0: x, 1: y), sense, low corner and high corner, segment, conductivity."""
    d = deck.discretization
    nodes, rows = np.array(deck.nodes), []
    for k, sg in enumerate(deck.segments):
        a, b = nodes[sg["a"]], nodes[sg["b"]]
        axis = 0 if abs(b[0] - a[0]) > abs(b[1] - a[1]) else 1
        sense = 1.0 if b[axis] > a[axis] else -1.0
        # the width direction is z x length
        across = sense if axis == 0 else -sense
        nw, nh = d["grids"][k] if "grids" in d else (d["nw"], d["nh"])
        wc, ws = _cells(sg["width"], nw, d.get("ratio", 1.0))
        hc, hs = _cells(sg["height"], nh, d.get("ratio", 1.0))
        for j in range(nh):
            for i in range(nw):
                mid, half = np.zeros(3), np.zeros(3)
                mid[axis], half[axis] = 0.5 * (a[axis] + b[axis]), 0.5 * abs(b[axis] - a[axis])
                mid[1 - axis], half[1 - axis] = a[1 - axis] + across * wc[i], 0.5 * ws[i]
                mid[2], half[2] = a[2] + hc[j], 0.5 * hs[j]
                rows.append((axis, sense, mid, half, k, sg["sigma"]))
    return rows


def _line_pairs(x, rho2):
    """x asinh(x / rho) - sqrt(x^2 + rho^2), even in x; the log(rho) part
    drops out of the second difference when the x share a sign."""
    r = torch.sqrt(x * x + rho2)
    return x.abs() * (torch.log(x.abs() + r) - 0.5 * torch.log(rho2)) - r


def _far(o, ha, hb, device):
    """Mutual integrals of parallel boxes apart: 5-point Gauss rules over both
    cross-sections, the two lengths in closed form.  o: centre offsets, ha and
    hb: half sizes, axis 0 along the length."""
    t, w = (torch.tensor(v, device=device) for v in np.polynomial.legendre.leggauss(5))
    out = []
    for k in range(0, len(o), 65536):
        O, A, B = (torch.tensor(np.asarray(v[k:k + 65536], dtype=np.float64), device=device) for v in (o, ha, hb))
        total = torch.zeros(len(O), dtype=torch.float64, device=device)
        for p in range(5):
            for q in range(5):
                # (cross axis 1, cross axis 2) of a by (p, q), of b by the grid
                dy = O[:, 1, None, None] + B[:, 1, None, None] * t[None, :, None] - A[:, 1, None, None] * t[p]
                dz = O[:, 2, None, None] + B[:, 2, None, None] * t[None, None, :] - A[:, 2, None, None] * t[q]
                rho2 = (dy * dy + dz * dz).clamp_min(1e-28)
                x, la, lb = O[:, 0, None, None], A[:, 0, None, None], B[:, 0, None, None]
                v = (_line_pairs(x + la + lb, rho2) - _line_pairs(x + la - lb, rho2)
                     - _line_pairs(x - la + lb, rho2) + _line_pairs(x - la - lb, rho2))
                total += w[p] * w[q] * (v * (w[None, :, None] * w[None, None, :])).sum((1, 2))
        out.append((total / 16.0).cpu().numpy())
    return np.concatenate(out) if out else np.zeros(0)


def _near(o, ha, hb):
    """The same integrals of touching, overlapping or close boxes: the
    64-term antiderivative (Hoer and Love 1965) in extended precision."""
    ld = np.longdouble
    o, ha, hb = (np.asarray(v, dtype=ld) for v in (o, ha, hb))

    def term(x, y, z):
        x2, y2, z2 = x * x, y * y, z * z
        r = np.sqrt(x2 + y2 + z2)

        def lg(u, a2, b2):
            c = a2 + b2
            ok = c > 0
            # log((u + r) / sqrt(c)) as an odd function of u
            v = np.log(np.where(ok, (np.abs(u) + r) / np.sqrt(np.where(ok, c, 1)), 1))
            return np.where(ok, np.sign(u) * v, 0)

        def at(a, b, c):
            d = c * r
            ok = d != 0
            return np.where(ok, np.arctan(a * b / np.where(ok, d, 1)), 0)

        y4, z4, x4 = y2 * y2, z2 * z2, x2 * x2
        return ((y2 * z2 / 4 - y4 / 24 - z4 / 24) * x * lg(x, y2, z2)
                + (x2 * z2 / 4 - x4 / 24 - z4 / 24) * y * lg(y, x2, z2)
                + (x2 * y2 / 4 - x4 / 24 - y4 / 24) * z * lg(z, x2, y2)
                + (x4 + y4 + z4 - 3 * (x2 * y2 + y2 * z2 + z2 * x2)) * r / 60
                - x * y * z2 * z / 6 * at(x, y, z) - x * y2 * y * z / 6 * at(x, z, y)
                - x2 * x * y * z / 6 * at(y, z, x))

    total = np.zeros(len(o), dtype=ld)
    corners = [(1, 1), (1, -1), (-1, 1), (-1, -1)]
    for sx, tx in corners:
        for sy, ty in corners:
            for sz, tz in corners:
                sign = sx * tx * sy * ty * sz * tz
                total += sign * term(o[:, 0] + sx * ha[:, 0] + tx * hb[:, 0], o[:, 1] + sy * ha[:, 1] + ty * hb[:, 1],
                                     o[:, 2] + sz * ha[:, 2] + tz * hb[:, 2])
    area = 16 * ha[:, 1] * ha[:, 2] * hb[:, 1] * hb[:, 2]
    return np.asarray(total / area, dtype=np.float64)


def _inductance(bars, device):
    n = len(bars)
    axis = np.array([b[0] for b in bars])
    sense = np.array([b[1] for b in bars])
    mid = np.array([b[2] for b in bars])
    half = np.array([b[3] for b in bars])
    L = np.zeros((n, n))
    mix = np.array([1000003, 10007, 998244353, 7368787, 15485863, 32452843, 49979687, 67867967, 86028121],
                   dtype=np.int64)
    for ax in (0, 1):
        of = np.nonzero(axis == ax)[0]
        i, j = (of[v] for v in np.triu_indices(len(of)))
        order = [ax, 1 - ax, 2]
        o, ha, hb = (mid[j] - mid[i])[:, order], half[i][:, order], half[j][:, order]
        # a deck repeats its offsets: integrate the distinct ones (to 1e-13 m)
        with np.errstate(over="ignore"):
            key = (np.round(np.hstack([np.abs(o), ha, hb]) / 1e-13).astype(np.int64) * mix).sum(1)
        _, first, back = np.unique(key, return_index=True, return_inverse=True)
        o, ha, hb = o[first], ha[first], hb[first]
        gap = np.linalg.norm(np.maximum(np.abs(o) - ha - hb, 0.0), axis=1)
        near = gap < 6.0 * np.maximum(ha[:, 1:].max(1), hb[:, 1:].max(1))
        v = np.empty(len(o))
        v[near] = _near(o[near], ha[near], hb[near])
        v[~near] = _far(o[~near], ha[~near], hb[~near], device)
        v = v[np.asarray(back).reshape(-1)] * sense[i] * sense[j] * (MU0 / (4.0 * math.pi))
        L[i, j] = v
        L[j, i] = v
    return L


def _nodal(deck, frequencies, currents=False):
    """Z between the ports (and the branch currents of 1 A into the first) by
    nodal analysis on the branch impedances R + jw L."""
    device = "cuda" if torch.cuda.is_available() else "cpu"
    bars = _bars(deck)
    n, ground = len(bars), len(deck.nodes) - 1
    area = np.array([4.0 * b[3][1 - b[0]] * b[3][2] for b in bars])
    length = np.array([2.0 * b[3][b[0]] for b in bars])
    R = length / (np.array([b[5] for b in bars]) * area)
    L = torch.tensor(_inductance(bars, device), device=device)
    inc = np.zeros((n, len(deck.nodes)))
    for k, b in enumerate(bars):
        sg = deck.segments[b[4]]
        inc[k, sg["a"]], inc[k, sg["b"]] = 1.0, -1.0
    inject = np.zeros((len(deck.nodes), len(deck.ports)))
    for k, (a, b) in enumerate(deck.ports):
        inject[a, k] += 1.0
        inject[b, k] -= 1.0
    A = torch.tensor(np.delete(inc, ground, 1), device=device, dtype=torch.complex128)
    J = torch.tensor(np.delete(inject, ground, 0), device=device, dtype=torch.complex128)
    Rd = torch.diag(torch.tensor(R, device=device))
    zs, flows = [], []
    for f in frequencies:
        Zb = torch.complex(Rd, 2.0 * math.pi * f * L)
        Y = torch.linalg.solve(Zb, A)
        v = torch.linalg.solve(A.T @ Y, J)
        zs.append((J.T @ v).cpu().numpy())
        if currents:
            flows.append((Y @ v[:, 0]).cpu().numpy())
    if not currents:
        return np.array(zs)
    segment = np.array([b[4] for b in bars])
    out = []
    for i in flows:
        density, power = np.abs(i) / area, 0.5 * np.abs(i) ** 2 * R
        sums = np.zeros(len(deck.segments), dtype=np.complex128)
        np.add.at(sums, segment, i)
        out.append({"current": i, "density": density, "power": power, "segment_current": sums,
                    "segment_power": np.bincount(segment, power, len(deck.segments)),
                    "peak_density": np.array([density.max()])})
    return out


def exact(case, seed):
    kind = case["kind"]
    if kind in ("solve", "sweep") and _filaments(case) <= EXACT_FILAMENTS:
        return _nodal(_deck(case, seed), _frequencies(case))
    if kind == "currents" and _filaments(case) <= EXACT_FILAMENTS:
        return _nodal(_deck(case, seed), _frequencies(case), currents=True)
    if kind == "batch":
        # the smaller members of the batch, up to 1,500 filaments in all
        out, room = [], 1500
        for d in _batch_decks(case, seed):
            n = len(d.segments) * d.discretization["nw"] * d.discretization["nh"]
            out.append(None if n > room else _nodal(d, _frequencies(case)))
            room -= n if n <= room else 0
        return out
    # The gradient, the general-position matrix (defined by its sampled
    # filaments) and the systems of 5,000 filaments and more take minutes.
    return None
