"""The pivoted panel's two cluster forms (slices in shared memory, slices in
device memory) on panels whose later rows leave CTAs of a cluster short or
without any, as the last panels of a factorization do: the same bits in FP64,
where a tie between two currents must fall the same way in both, and each
form's pivots and entries against numpy in FP64 and FP32.

Tolerances: at most 128 rank-1 updates of rounding u with a growth below 10:
128 x 10 u of the largest entry, 1.5e-4 in FP32 and 3e-13 in FP64.  A pivot
may differ from numpy's only among candidates that near: the pivot chosen is
as large as the largest up to that rounding, and numpy follows it."""
import ctypes

import numpy as np
import pytest

from fasterhenry_b200 import _native as N

pytestmark = pytest.mark.gpu

# the order plans 16 CTAs a matrix at most; k0 leaves 2 to 140 rows to them
CASES = [(900, 1, 896, 4), (900, 3, 832, 64), (1000, 1, 960, 40), (130, 2, 128, 2), (200, 4, 128, 64),
         (900, 4, 0, 64), (1024, 1, 884, 64)]


def factor(a, k0, nb, single, resident):
    count, m, _ = a.shape
    dev = np.ascontiguousarray(a.transpose(0, 2, 1))  # column-major
    piv = np.zeros((count, m), dtype=np.int32)
    sing = np.zeros(count, dtype=np.int32)
    info = N.ErrorInfo()
    ip = lambda v: v.ctypes.data_as(ctypes.POINTER(ctypes.c_int32))
    st = N.load().fh_test_panel_form(dev.ctypes.data_as(N.c_double_p), m, count, k0, nb, single, resident, ip(piv),
                                     ip(sing), ctypes.byref(info))
    assert st == N.OK, N.last_error()
    assert not sing.any()
    return dev.transpose(0, 2, 1), piv[:, k0:k0 + nb]


def check(a, got, piv, k0, nb, tol):
    """numpy's elimination with the pivots that were chosen."""
    a = a.copy()
    w = slice(k0, k0 + nb)
    for j in range(k0, k0 + nb):
        size = np.abs(a[j:, j].real) + np.abs(a[j:, j].imag)
        p = piv[j - k0]
        assert size[p - j] >= size.max() - tol * np.abs(a[k0:, w]).max()
        a[[j, p], w] = a[[p, j], w]
        a[j + 1:, j] /= a[j, j]
        a[j + 1:, j + 1:k0 + nb] -= np.outer(a[j + 1:, j], a[j, j + 1:k0 + nb])
    assert np.max(np.abs(got[k0:, w] - a[k0:, w])) <= tol * np.max(np.abs(a[k0:, w]))


@pytest.mark.parametrize("m,count,k0,nb", CASES)
def test_forms_agree_bit_for_bit_in_fp64(fh, m, count, k0, nb):
    rng = np.random.default_rng(m + count)
    a = rng.standard_normal((count, m, m)) + 1j * rng.standard_normal((count, m, m))
    a[:, (k0 + m - 1) // 2] = a[:, m - 1].conj()  # two candidates of equal size in the first column
    want, want_piv = factor(a, k0, nb, 0, 0)
    for _ in range(3):
        got, piv = factor(a, k0, nb, 0, 1)
        assert np.array_equal(piv, want_piv) and np.array_equal(got, want)


@pytest.mark.parametrize("resident", [0, 1])
@pytest.mark.parametrize("single", [0, 1])
@pytest.mark.parametrize("m,count,k0,nb", CASES + [(464, 8, 384, 80), (464, 8, 0, 128), (900, 2, 768, 128)])
def test_each_form_matches_numpy(fh, m, count, k0, nb, single, resident):
    rng = np.random.default_rng(m + nb)
    a = rng.standard_normal((count, m, m)) + 1j * rng.standard_normal((count, m, m))
    if single:
        a = a.astype(np.complex64).astype(np.complex128)
    got, piv = factor(a, k0, nb, single, resident)
    for f in range(min(count, 2)):
        check(a[f], got[f], piv[f], k0, nb, 1.5e-4 if single else 3e-13)


def test_a_plan_without_a_cluster(fh):
    """A plan of one CTA a matrix is no cluster: neither form, and the same
    result whichever is asked for."""
    rng = np.random.default_rng(5)
    a = rng.standard_normal((2, 60, 60)) + 1j * rng.standard_normal((2, 60, 60))
    want, piv = factor(a, 0, 60, 0, 0)
    got, piv2 = factor(a, 0, 60, 0, 1)
    assert np.array_equal(piv, piv2) and np.array_equal(got, want)
    check(a[0], got[0], piv[0], 0, 60, 3e-13)
