"""Many equal items through the batched kernel, alone and by groups of CTAs,
with every diagonal tile full (the inverse of its factor takes the tile's own
place) and with the ports inside the last tile: each item's sums run in a
fixed order, so all of them end in the same bits, and match numpy.

Tolerance: as for the batched kernel's other tests, 64 x 2.2e-16 x 20 x
sqrt(m) < 1e-11 for m <= 700."""
import numpy as np
import pytest

from test_gpu_batch_tiles import solve, spd

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("config,edge", [(0, 32), (1, 32), (2, 64), (3, 64)])
@pytest.mark.parametrize("tiles", [1, 2, 5])
@pytest.mark.parametrize("inside", [False, True])
def test_equal_items_have_equal_bits(fh, config, edge, tiles, inside):
    p = 3 if inside else edge
    m = tiles * edge - (p if inside else 0)
    rng = np.random.default_rng(m)
    r, l = spd(rng, m + p), spd(rng, m + p)
    z, failed = solve(r, l, m, p, np.full(900, 0.7), config, 300)
    assert not failed.any()
    assert np.array_equal(z, np.broadcast_to(z[0], z.shape))
    a = r + 0.7j * l
    want = a[m:, m:] - a[m:, :m] @ np.linalg.solve(a[:m, :m], a[:m, m:])
    assert np.max(np.abs(z[0] - want)) <= 1e-11 * np.max(np.abs(want))
