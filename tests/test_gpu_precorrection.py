"""The precorrection cancels the grid's own approximation of every near pair:
the product's column L e_i must return the exact partial inductance on the
near pairs, whatever the grid contributes there.  Rows that take the grid
potential over their partners' hull (short filaments, flat and deep hulls,
hulls of several slabs), rows that go pair by pair (filaments as long as the
deck), small and large stencils.

The cancelled terms are sums of at most 1e5 products of either sign with an
absolute sum below 10 times the largest entry, and the convolution over P
points adds u log2(P): 1e-12 of the largest entry bounds both."""
import numpy as np
import pytest

from fasterhenry_b200 import fixtures as F

pytestmark = pytest.mark.gpu


def flat(runs):
    return F.scaling_meander(runs)


def cloud(manhattan):
    return F.cloud_deck(220, manhattan, 7)


def long_and_short():
    """A few bars across the whole deck among short ones."""
    deck = F.cloud_deck(150, True, 9)
    nodes, segs = list(deck.nodes), list(deck.segments)
    side = F.cloud_side(150)
    for k in range(6):
        y = side * (k + 0.5) / 6
        nodes += [(-2 * side, y, 0.3 * side), (3 * side, y, 0.3 * side)]
        segs.append(F.segment(len(nodes) - 2, len(nodes) - 1, 0.1e-3, 0.05e-3))
    return F.Deck(nodes, segs, [], F.uniform(1, 1), "long_and_short")


@pytest.mark.parametrize("deck", [flat(7), cloud(True), cloud(False), long_and_short()],
                         ids=["flat", "manhattan", "general", "long"])
@pytest.mark.parametrize("order,radius", [(2, 3.0), (5, 8.0), (7, 14.0)])
def test_near_pairs_come_out_exact(fh, deck, order, radius):
    fil, _ = fh.discretize(fh.Geometry.from_deck(deck), deck.discretization)
    n = len(fil)
    exact = fh.partial_inductance_matrix(fil)
    with fh.PfftOperator(fil, fh.PfftParams(near_field_radius=radius, interpolation_order=order)) as op:
        h = op.stats()["grid_spacing"]
        off, cols = fh.near_pairs(fil, radius * h)
        worst = 0.0
        picked = range(0, n, max(1, n // 40))
        for i in picked:
            x = np.zeros(n)
            x[i] = 1.0
            column = op.apply(x)
            near = cols[off[i]:off[i + 1]]
            assert i in near
            worst = max(worst, np.max(np.abs(column[near] - exact[near, i])))
    assert worst <= 1e-12 * np.max(np.abs(exact)), worst / np.max(np.abs(exact))
