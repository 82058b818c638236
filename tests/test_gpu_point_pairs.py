"""Point-quadrature pairs whose terms a warp shares (512 terms and more)
against those that a thread sums alone: pairs across the whole range of costs
match the oracle, and a pair's value does not depend on the list it is in."""
import numpy as np
import pytest

from fasterhenry_b200 import fixtures as F

pytestmark = pytest.mark.gpu


def bars(kind, count=40):
    """Bars of one frame (parallel), of one frame but unequal sizes, or in
    general position, at distances from a fraction of their length (orders up
    to 20 along it) to a hundred lengths."""
    rng = np.random.default_rng(len(kind))
    nodes, segs = [], []
    for k in range(count):
        length = 1e-3 if kind == "equal" else 1e-3 * (0.3 + rng.random())
        at = np.array([0.2e-3 * rng.random(), 0.45e-3 * 1.22 ** k, 0.1e-3 * rng.random()])
        d = np.array([1.0, 0.0, 0.0])
        if kind == "general":
            d = rng.standard_normal(3)
            d /= np.linalg.norm(d)
        w, h = (0.1e-3, 0.06e-3) if kind == "equal" else 1e-4 * (0.4 + rng.random(2))
        nodes += [tuple(at - 0.5 * length * d), tuple(at + 0.5 * length * d)]
        segs.append(F.segment(2 * k, 2 * k + 1, float(w), float(h)))
    return F.Deck(nodes, segs, [], F.uniform(1, 1), kind)


@pytest.mark.parametrize("kind", ["equal", "parallel", "general"])
def test_costs_across_the_threshold_match_the_oracle(fh, oracle, kind):
    """1e-10 relative per entry, the fill's tolerance against the oracle."""
    deck = bars(kind)
    fil, _ = fh.discretize(fh.Geometry.from_deck(deck), deck.discretization)
    got, ref = fh.partial_inductance_matrix(fil), oracle.fill(fil)
    zero = ref == 0.0
    assert np.array_equal(got[zero], ref[zero])
    assert np.max(np.abs(got[~zero] - ref[~zero]) / np.abs(ref[~zero])) < 1e-10


@pytest.mark.parametrize("kind", ["equal", "general"])
def test_a_pairs_value_does_not_depend_on_its_list(fh, kind):
    deck = bars(kind)
    fil, _ = fh.discretize(fh.Geometry.from_deck(deck), deck.discretization)
    whole = fh.partial_inductance_matrix(fil)
    for i, j in [(0, 1), (0, 2), (1, 3), (0, 9), (4, 30), (20, 39)]:
        assert fh.mutual_inductance(fil[i], fil[j]) == whole[i, j]
