"""One panel of the pivoted FP64 factorization against numpy: orders whose
slices end with, before and after a CTA's 64 rows, the first and a later
panel, narrow panels, one matrix (a cluster of up to 16 CTAs, slices in shared
memory up to 168 rows), several, and many whose slices stay in device memory.

Tolerances: random entries have no ties, so the interchanges must be numpy's;
the entries carry at most 64 rank-1 updates of rounding 2.2e-16 each, with a
growth below 10 for these sizes: 1e-12 of the largest."""
import ctypes

import numpy as np
import pytest

from fasterhenry_b200 import _native as N

pytestmark = pytest.mark.gpu


def factor(a, k0, nb):
    count, m, _ = a.shape
    dev = np.ascontiguousarray(a.transpose(0, 2, 1))  # column-major
    piv = np.zeros((count, m), dtype=np.int32)
    sing = np.zeros(count, dtype=np.int32)
    info = N.ErrorInfo()
    ip = lambda v: v.ctypes.data_as(ctypes.POINTER(ctypes.c_int32))
    st = N.load().fh_test_panel(dev.ctypes.data_as(N.c_double_p), m, count, k0, nb, ip(piv), ip(sing),
                                ctypes.byref(info))
    assert st == N.OK, N.last_error()
    return dev.transpose(0, 2, 1), piv, sing


def panel(a, k0, nb):
    a = a.copy()
    piv = []
    for j in range(k0, k0 + nb):
        p = j + int(np.argmax(np.abs(a[j:, j].real) + np.abs(a[j:, j].imag)))
        piv.append(p)
        a[[j, p], k0:k0 + nb] = a[[p, j], k0:k0 + nb]
        a[j + 1:, j] /= a[j, j]
        a[j + 1:, j + 1:k0 + nb] -= np.outer(a[j + 1:, j], a[j, j + 1:k0 + nb])
    return a, np.array(piv)


@pytest.mark.parametrize("m,count,k0,nb", [(1, 1, 0, 1), (5, 1, 0, 5), (64, 2, 0, 64), (65, 2, 0, 64), (70, 1, 64, 6),
                                           (130, 3, 0, 64), (200, 1, 64, 64), (200, 4, 128, 64), (333, 1, 0, 17),
                                           (900, 4, 0, 64), (900, 2, 832, 64), (1025, 1, 0, 64), (2400, 1, 0, 64),
                                           (2700, 1, 0, 64), (640, 30, 0, 64)])
def test_panel_matches_numpy(fh, m, count, k0, nb):
    rng = np.random.default_rng(m + count)
    a = rng.standard_normal((count, m, m)) + 1j * rng.standard_normal((count, m, m))
    got, piv, sing = factor(a, k0, nb)
    assert not sing.any()
    for f in range(min(count, 3)):
        want, want_piv = panel(a[f], k0, nb)
        assert np.array_equal(piv[f, k0:k0 + nb], want_piv)
        w = slice(k0, k0 + nb)
        assert np.max(np.abs(got[f][k0:, w] - want[k0:, w])) <= 1e-12 * np.max(np.abs(want[k0:, w]))
        assert np.array_equal(got[f][:, :k0], a[f][:, :k0]) and np.array_equal(got[f][:k0], a[f][:k0])


@pytest.mark.parametrize("m", [40, 200])
def test_ties_zero_columns_and_nan(fh, m):
    """The first of equal candidates; a zero column is flagged and keeps its
    diagonal; a column of NaN keeps its diagonal, too."""
    a = np.ones((3, m, m), dtype=np.complex128) + np.diag(np.arange(m))
    a[1, :, 0] = 0.0
    a[2, :, 0] = np.nan
    got, piv, sing = factor(a, 0, 32)
    assert list(sing) == [0, 1, 0]
    assert list(piv[:, 0]) == [0, 0, 0]
    want, want_piv = panel(a[0], 0, 32)
    assert np.array_equal(piv[0, :32], want_piv)
