"""Coordinate derivatives of parallel bars where the point rule is the more
accurate of the two that could take them: stout bars some four sides apart,
and thin ones nearly in one line, against a reference in extended precision.

Reference: Gauss rules of 12 nodes over both cross-sections (gaps of four
sides and more, or thin bars: converged to 1e-15) of the line integrals in
closed form.

Tolerance for the derivatives along and across the bars: the point rule's
orders meet 1e-8 for 1 / R, and one node more per axis is worth a further
(1 + 2 gap / side)^2, 50 at least here: 2e-10."""
import numpy as np
import pytest

from test_gpu_coordinate_gradient import Box

pytestmark = pytest.mark.gpu

UM = 1e-6
LD = np.longdouble


def derivatives(da, db, off):
    """dL/d(translation of a along x, along y) of boxes along x, off from a's
    centre to b's."""
    da, db, off = (np.asarray(v, dtype=LD) for v in (da, db, off))
    x, w = (v.astype(LD) for v in np.polynomial.legendre.leggauss(12))
    w /= w.sum()
    ya, za, yb, zb = np.meshgrid(x * da[1] / 2, x * da[2] / 2, off[1] + x * db[1] / 2, off[2] + x * db[2] / 2,
                                 indexing="ij")
    weight = np.einsum("i,j,k,l->ijkl", w, w, w, w)
    rho2 = (ya - yb) ** 2 + (za - zb) ** 2
    a, b = da[0] / 2, db[0] / 2

    def corners(f):  # int int f''(x' - x)
        return f(off[0] + b + a) - f(off[0] - b + a) - f(off[0] + b - a) + f(off[0] - b - a)
    along = corners(lambda t: -np.arcsinh(t / np.sqrt(rho2)))
    across = -(ya - yb) * corners(lambda t: np.sqrt(t * t + rho2)) / rho2
    return float((weight * along).sum()) * 1e-7, float((weight * across).sum()) * 1e-7


@pytest.mark.parametrize("da,db,off", [
    ((145.74, 56.61, 71.93), (66.07, 32.54, 63.89), (49.37, 200.48, 339.13)),
    ((92.69, 12.96, 34.62), (57.29, 32.64, 37.3), (-13.56, 32.43, 203.97)),
    ((112.37, 0.32, 0.3), (77.32, 0.67, 0.6), (-133.79, -0.001, 2.09)),
    ((240.37, 1.56, 1.05), (283.52, 2.44, 1.48), (360.62, -0.058, 6.39)),
    # where the panels' rule is better: thin bars apart
    ((120.0, 2.0, 1.0), (100.0, 1.5, 2.0), (30.0, 250.0, 40.0))])
def test_along_and_across(fh, da, db, off):
    da, db, off = (np.array(v) * UM for v in (da, db, off))
    boxes = [Box((0, 0, 0), (1, 0, 0), da), Box(off, (1, 0, 0), db)]
    dl, dp, _, _ = fh.coordinate_gradient(np.array([b.filament() for b in boxes]), [0, 1])
    want = derivatives(da, db, off)
    assert abs(dl[0, 1] - want[0]) <= 2e-10 * abs(want[0])
    assert abs(dp[0, 1] - want[1]) <= 2e-10 * abs(want[1])
