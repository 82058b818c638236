"""Mixed-precision sweeps of orders whose last 128-column block has few, some and
most of its rows, and of a single partial block: the diagonal blocks' factors
and inverses precondition the refinement, which has to converge in a few steps
to the FP64 sweep.

Tolerance: the refinement stops at corrections of 1e-12 of the solution; Z
follows within a small factor of that, 1e-9 is the sweeps' stated bound."""
import numpy as np
import pytest

from fasterhenry_b200 import fixtures as F

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("legs,nw,nh", [(1, 4, 1), (2, 5, 3), (4, 6, 2), (5, 4, 3), (7, 10, 2), (9, 8, 2), (11, 10, 3),
                                        # orders 128, 130, 132, 510, 512, 516
                                        (8, 3, 3), (5, 7, 2), (6, 4, 3), (15, 6, 3), (8, 11, 3), (6, 11, 4)])
def test_mixed_matches_fp64(fh, legs, nw, nh):
    deck = F.meander_legs(legs, nw=nw, nh=nh)
    freqs = [1e6, 1e8, 1e10]
    with fh.MeshSystem.assemble(fh.Geometry.from_deck(deck), deck.ports, deck.discretization) as s:
        want = s.sweep(freqs, fh.Precision.FP64)
        got = s.sweep(freqs, fh.Precision.MIXED_BF16X3)
    rel = np.max(np.abs(got.impedance_ohm - want.impedance_ohm) / np.abs(want.impedance_ohm))
    assert rel < 1e-9, rel
