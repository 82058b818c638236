"""The block products of the Krylov solver and the pFFT product's vector
pairs, at the sizes where their tiles end."""
import numpy as np
import pytest

from fasterhenry_b200 import fixtures as F

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 2, 63, 64, 65, 129, 640, 1025])
def test_basis_products_over_row_chunks_and_vector_groups(fh, n):
    """A dense complex system whose Krylov space passes one group of 8 basis
    vectors (and two of them) with fewer rows than chunks (64), as many, and
    tails.  A = 4 I + E with |E|_2 < 2 has a condition number below 3, so a
    relative residual of 1e-12 leaves an error below 3e-12."""
    rng = np.random.default_rng(n)
    e = rng.standard_normal((n, n)) + 1j * rng.standard_normal((n, n))
    a = 4.0 * np.eye(n) + 1.9 * e / np.linalg.norm(e, 2)
    b = rng.standard_normal(n) + 1j * rng.standard_normal(n)
    x, oc = fh.gmres_dense(a, b, params=fh.GmresParams(tolerance=1e-12, restart=100, max_iterations=500))
    want = np.linalg.solve(a, b)
    assert oc.converged
    assert n < 20 or oc.iterations > 16  # more than two groups of vectors
    assert np.linalg.norm(x - want) <= 3e-12 * np.linalg.norm(want)


@pytest.mark.parametrize("axes", [1, 2, 3])
@pytest.mark.parametrize("count", [1, 2, 3, 4, 5])
def test_products_of_several_vectors_equal_single_ones(fh, axes, count):
    """Vectors travel in pairs (an odd last one alone) over 1, 2 or 3 field
    components; each must come out as from its own product.  The sums are the
    same terms, the two transforms of a pair share one complex grid: the
    difference is FP64 rounding, u log2(P) < 1e-14 of the largest entry of
    the pair."""
    nodes, segs = F.cloud_bars(150, 4e-3, True, 31)
    keep = []
    for k in range(len(segs)):
        d = np.subtract(nodes[2 * k + 1], nodes[2 * k])
        if int(np.argmax(np.abs(d))) < axes:
            keep.append(k)
    deck_nodes = [nodes[i] for k in keep for i in (2 * k, 2 * k + 1)]
    deck_segs = [dict(segs[k], a=2 * q, b=2 * q + 1) for q, k in enumerate(keep)]
    deck = F.Deck(deck_nodes, deck_segs, [], F.uniform(1, 1), "cloud")
    fil, _ = fh.discretize(fh.Geometry.from_deck(deck), deck.discretization)
    rng = np.random.default_rng(count)
    x = rng.standard_normal((count, len(fil)))
    with fh.PfftOperator(fil) as op:
        together = op.apply(x)
        single = np.array([op.apply(v) for v in x])
    assert np.max(np.abs(together - single)) <= 1e-13 * np.max(np.abs(single))
