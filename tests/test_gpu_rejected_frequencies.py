"""Sweeps whose list holds frequencies that the elimination without
interchanges rejects among others that it takes: the rejected ones are redone
with interchanges and end in their own places.

The deck's conductivity is so large that its resistances are near 1e-155 ohm.
At zero frequency the squared modulus of a pivot, near 1e-310, has no finite
reciprocal, and the elimination without interchanges rejects it; at 1 GHz the
same system is an ordinary one.  The direct-current impedance is that of the
same deck of copper times the ratio of the conductivities.

Tolerances: a squared pivot of 1e-311 or more carries a rounding of 5e-324 /
1e-311 = 5e-13, once per pivot and once per solve with it: 1e-9 for the few
hundred pivots here.  At 1 GHz 1e-10, as for the other sweeps, of the deck
against the oracle's on the same deck."""
import dataclasses

import numpy as np
import pytest

from fasterhenry_b200 import fixtures as F

from test_gpu_ldlt import solve

pytestmark = pytest.mark.gpu

SIGMA = 1e162
FREQS = [1e9, 0.0, 3e9, 0.0, 0.0, 2e9]


def decks(legs, nw):
    """The deck of copper and the one of SIGMA, two ports."""
    copper = F.meander(legs, 1e-3, 40e-6, 20e-6, 5e-6, F.uniform(nw, 2))
    last = len(copper.nodes) - 1
    copper.ports = [(0, last // 2), (last // 2, last)]
    extreme = dataclasses.replace(copper, segments=[dict(s, sigma=SIGMA) for s in copper.segments])
    return copper, extreme


def expected(oracle, copper, extreme):
    dc = oracle.System(copper).impedance(0.0) * (F.COPPER / SIGMA)
    system = oracle.System(extreme)
    return [system.impedance(f) if f else dc for f in FREQS]


def check(got, want):
    for z, w, f in zip(got, want, FREQS):
        assert np.max(np.abs(z - w)) <= (1e-10 if f else 1e-9) * np.max(np.abs(w)), f


# one panel, several, and with the panels on a stream of their own
@pytest.mark.parametrize("legs,nw", [(2, 3), (5, 4), (12, 8)])
def test_sweep(fh, oracle, legs, nw):
    copper, extreme = decks(legs, nw)
    with fh.MeshSystem.assemble(fh.Geometry.from_deck(extreme), extreme.ports, extreme.discretization) as s:
        z = s.sweep(FREQS, fh.Precision.FP64).impedance_ohm
        again = s.sweep(FREQS[::-1], fh.Precision.FP64).impedance_ohm
        r, l = s.mesh_matrices()
        _, _, rejected = solve(r, l, len(r) - 2, 2, 2 * np.pi * np.array(FREQS))
    assert list(rejected) == [f == 0.0 for f in FREQS]
    check(z, expected(oracle, copper, extreme))
    check(again[::-1], expected(oracle, copper, extreme))


def test_batch_of_ordinary_and_rejected_items(fh, oracle):
    copper, extreme = decks(5, 4)
    systems = [fh.MeshSystem.assemble(fh.Geometry.from_deck(d), d.ports, d.discretization)
               for d in (copper, extreme, copper)]
    try:
        results = fh.batch_sweep(systems, [FREQS] * 3, fh.Precision.MIXED_BF16X3)
    finally:
        for s in systems:
            s.close()
    plain = oracle.System(copper)
    check(results[1].impedance_ohm, expected(oracle, copper, extreme))
    for k in (0, 2):
        check(results[k].impedance_ohm, [plain.impedance(f) for f in FREQS])


def test_gradient(fh):
    """The gradient's loop currents come from the redone solve; at zero
    frequency it goes as 1 / conductivity."""
    copper, extreme = decks(5, 4)
    params = [fh.Param("width", 1), fh.Param("thickness", 4), fh.Param("x", 3)]
    out = []
    for deck in (copper, extreme):
        with fh.MeshSystem.assemble(fh.Geometry.from_deck(deck), deck.ports, deck.discretization) as s:
            out.append(s.gradient(0.0, params))
    scale = F.COPPER / SIGMA
    for got, want in ((out[1].impedance_ohm, out[0].impedance_ohm), (out[1].gradient, out[0].gradient)):
        assert np.max(np.abs(got - want * scale)) <= 1e-9 * np.max(np.abs(want)) * scale
