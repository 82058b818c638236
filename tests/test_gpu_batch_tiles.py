"""The batched kernel's factorization (fh_batchsolve.cu) in each of its tile
configurations, at the ends of the tiles: orders that leave no padding, one
row of it or all but one, ports that fit the last tile, fill it and take tiles
of their own; against numpy.

Tolerance: that of the factorization without interchanges on matrices with
kappa <= 20, 64 x 2.2e-16 x 20 x sqrt(m) < 1e-11 for m <= 700."""
import ctypes

import numpy as np
import pytest

from fasterhenry_b200 import _native as N

pytestmark = pytest.mark.gpu


def spd(rng, n):
    q, _ = np.linalg.qr(rng.standard_normal((n, n)))
    a = (q * np.linspace(1.0, 10.0, n)) @ q.T
    return 0.5 * (a + a.T)


def solve(r, l, m, p, omega, config, grouped=0):
    r, l = np.asfortranarray(r), np.asfortranarray(l)
    w = np.ascontiguousarray(omega, dtype=np.float64)
    z = np.zeros((len(omega), p, p), dtype=np.complex128)
    failed = np.zeros(len(omega), dtype=np.int32)
    info = N.ErrorInfo()
    dp = lambda a: a.ctypes.data_as(N.c_double_p)
    st = N.load().fh_test_batch_solve(dp(r), dp(l), m, p, dp(w), len(omega), config, grouped, dp(z),
                                      failed.ctypes.data_as(ctypes.POINTER(ctypes.c_int32)), ctypes.byref(info))
    assert st == N.OK, N.last_error()
    return z, failed


@pytest.mark.parametrize("grouped", [0, 3])  # the fourth then by a CTA alone, after them
@pytest.mark.parametrize("config", range(4))
@pytest.mark.parametrize("p", [1, 2, 31, 32, 70])
@pytest.mark.parametrize("m", [0, 1, 30, 31, 32, 33, 62, 63, 64, 65, 126, 127, 128, 300, 577])
def test_matches_numpy(fh, m, p, config, grouped):
    rng = np.random.default_rng(100 * m + p)
    r, l = spd(rng, m + p), spd(rng, m + p)
    omega = [0.0, 0.3, 1.0, 40.0]
    z, failed = solve(r, l, m, p, omega, config, grouped)
    assert not failed.any()
    for k, w in enumerate(omega):
        a = r + 1j * w * l
        want = a[m:, m:] - a[m:, :m] @ np.linalg.solve(a[:m, :m], a[:m, m:])
        assert np.max(np.abs(z[k] - want)) <= 1e-11 * np.max(np.abs(want))
        assert np.array_equal(z[k], z[k].T)
        assert w != 0.0 or not z[k].imag.any()


@pytest.mark.parametrize("grouped", [0, 1])
@pytest.mark.parametrize("config", range(4))
@pytest.mark.parametrize("m", [40, 64, 150])
def test_rejects_what_needs_pivoting(fh, m, config, grouped):
    """A tiny or zero pivot against O(1) couplings, and a NaN; the items that
    follow in the same CTAs are not touched."""
    rng = np.random.default_rng(m)
    good_r, good_l = spd(rng, m + 1), spd(rng, m + 1)
    for where in [0, m - 2]:
        for value in [1e-9, 0.0, np.nan]:
            r = good_r.copy()
            r[where, :] = r[:, where] = 0.0
            r[where, m - 1] = r[m - 1, where] = 1.0
            r[where, where] = value
            z, failed = solve(r, np.zeros_like(r), m, 1, [0.0, 1.0], config, grouped)
            assert failed.all(), (where, value)
    z, failed = solve(good_r, good_l, m, 1, np.linspace(0.0, 2.0, 700), config, 350 * grouped)
    assert not failed.any() and np.isfinite(z).all()
