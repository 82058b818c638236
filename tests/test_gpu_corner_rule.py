"""The orthogonal pairs' corner rule where a corner coordinate is zero or
changes sign, against the oracle's bar integral of the two boxes (1e-9, as
the other orthogonal pairs)."""
import numpy as np
import pytest

from test_gpu_coordinate_gradient import MU0_4PI, UM, Box, device_d

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("along", [0.0, 125.0, -125.0, 300.0])   # b's centre along its own length, um
@pytest.mark.parametrize("across", [0.0, 150.0, 170.0])          # and along a's
@pytest.mark.parametrize("up", [6.0, 18.0])
def test_corner_coordinates_of_every_sign(fh, oracle, along, across, up):
    """b runs along y above a (along x): its ends lie on a's axis (a zero
    corner), on either side of it, or past its end."""
    a = Box([0, 0, 0], [1, 0, 0], [300 * UM, 2 * UM, 1 * UM])
    b = Box([across * UM, along * UM, up * UM], [0, 1, 0], [250 * UM, 2 * UM, 1 * UM])
    D = device_d(fh, [a, b], [0, 1])
    ext = [sum(abs(ax @ bx) * d for bx, d in zip([b.l, b.w, b.h], b.dims)) for ax in [a.l, a.w, a.h]]
    off = [ax @ (b.c - a.c) for ax in [a.l, a.w, a.h]]
    v = oracle.aligned_quadrature([a.dims[0], ext[0]], [a.dims[1], ext[1]], [a.dims[2], ext[2]], off)
    k = MU0_4PI / (a.dims[1] * a.dims[2] * b.dims[1] * b.dims[2])
    want = k * (np.cross([0, 0, 1], a.l) @ b.l) * v
    assert abs(D[3][0, 1] - want) <= 1e-9 * abs(want), (D[3][0, 1], want)
    assert abs(D[3][1, 0] + want) <= 1e-9 * abs(want), (D[3][1, 0], -want)
