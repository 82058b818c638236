"""The FP64 factorization without interchanges (fh_ldlt.cu) on mesh systems
R + j w L with both parts positive definite, at the ends of its 64-column
panels and 64-row tiles, against numpy; and its rejection of systems that
elimination without pivoting does not suit.

Tolerance: the relative error of a backward-stable solve is at most about
m u kappa.  The test matrices have kappa(R), kappa(L) <= 10, so kappa of R +
j w L is at most 20: 64 x 2.2e-16 x 20 x sqrt(m) < 1e-11 for m <= 700."""
import ctypes

import numpy as np
import pytest

from fasterhenry_b200 import _native as N

pytestmark = pytest.mark.gpu


def spd(rng, n):
    q, _ = np.linalg.qr(rng.standard_normal((n, n)))
    a = (q * np.linspace(1.0, 10.0, n)) @ q.T
    return 0.5 * (a + a.T)


def solve(r, l, m, p, omega):
    count = len(omega)
    r, l = np.asfortranarray(r), np.asfortranarray(l)
    w = np.ascontiguousarray(omega, dtype=np.float64)
    z = np.zeros((count, p, p), dtype=np.complex128)
    x = np.zeros((count, p, m), dtype=np.complex128)
    failed = np.zeros(count, dtype=np.int32)
    info = N.ErrorInfo()
    dp = lambda a: a.ctypes.data_as(N.c_double_p)
    st = N.load().fh_test_mesh_solve(dp(r), dp(l), m, p, dp(w), count, dp(z), dp(x),
                                     failed.ctypes.data_as(ctypes.POINTER(ctypes.c_int32)), ctypes.byref(info))
    assert st == N.OK, N.last_error()
    return z, x, failed


@pytest.mark.parametrize("m", [1, 2, 15, 16, 17, 31, 63, 64, 65, 127, 128, 129, 200, 321, 640])
@pytest.mark.parametrize("p", [1, 3, 70])
def test_matches_numpy(fh, m, p):
    rng = np.random.default_rng(100 * m + p)
    r, l = spd(rng, m + p), spd(rng, m + p)
    omega = [0.0, 0.3, 1.0, 40.0]
    z, x, failed = solve(r, l, m, p, omega)
    assert not failed.any()
    for k, w in enumerate(omega):
        a = r + 1j * w * l
        want_x = np.linalg.solve(a[:m, :m], a[:m, m:])
        want_z = a[m:, m:] - a[m:, :m] @ want_x
        assert np.max(np.abs(x[k].T - want_x)) <= 1e-11 * np.max(np.abs(want_x))
        assert np.max(np.abs(z[k] - want_z)) <= 1e-11 * np.max(np.abs(want_z))
        assert np.array_equal(z[k], z[k].T)
        assert w != 0.0 or not z[k].imag.any()


@pytest.mark.parametrize("m,count", [(65, 24), (130, 140), (256, 80), (257, 30), (321, 24), (577, 48), (640, 40)])
@pytest.mark.parametrize("p", [1, 70])
def test_groups_of_panels(fh, m, p, count):
    """Enough matrices for groups of two and of four panels (partial ones at the
    end, and orders on both sides of the panels' own stream)."""
    rng = np.random.default_rng(10 * m + p)
    r, l = spd(rng, m + p), spd(rng, m + p)
    omega = np.linspace(0.0, 3.0, count)
    z, x, failed = solve(r, l, m, p, omega)
    assert not failed.any()
    for k in [0, 1, count // 2, count - 1]:
        a = r + 1j * omega[k] * l
        want_x = np.linalg.solve(a[:m, :m], a[:m, m:])
        want_z = a[m:, m:] - a[m:, :m] @ want_x
        assert np.max(np.abs(x[k].T - want_x)) <= 1e-11 * np.max(np.abs(want_x))
        assert np.max(np.abs(z[k] - want_z)) <= 1e-11 * np.max(np.abs(want_z))


@pytest.mark.parametrize("m", [40, 64, 150])
def test_rejects_what_needs_pivoting(fh, m):
    """Rows whose elimination grows: a tiny leading pivot against O(1)
    couplings (inside the first panel, and in the second one), an exactly zero
    pivot, and a NaN; a good matrix in the same batch is not touched."""
    rng = np.random.default_rng(m)
    good_r, good_l = spd(rng, m + 1), spd(rng, m + 1)
    for where in [0, m - 2]:
        for value in [1e-9, 0.0, np.nan]:
            r = good_r.copy()
            r[where, :] = r[:, where] = 0.0
            r[where, m - 1] = r[m - 1, where] = 1.0
            r[where, where] = value
            z, x, failed = solve(r, np.zeros_like(r), m, 1, [0.0, 1.0])
            assert failed.all(), (where, value)
    z, x, failed = solve(good_r, good_l, m, 1, [0.0, 1.0])
    assert not failed.any()
