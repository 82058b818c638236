"""The grid convolution's transforms over axis lengths that use every register
radix (1 to 16), one to five stages, and lines that do not fill a tile, on
each axis (strided axes 0 and 1, contiguous axis 2), against numpy's FFT.

Tolerances: a transform of length m in precision u has a relative error of
about u log2(m) in the 2-norm; forward and inverse over three axes of a torus
of P points give 2 u log2(P), at most 2 x 6e-8 x 15 = 1.8e-6 in FP32 and
3e-15 in FP64 here; the potentials' max-norm is within a small factor of
their 2-norm per point, so 4e-6 and 1e-12 are the bounds."""
import numpy as np
import pytest

from test_gpu_fftconv import reference

pytestmark = pytest.mark.gpu

LENGTHS = [1, 2, 3, 4, 5, 6, 8, 9, 10, 12, 15, 16, 18, 25, 27, 32, 125, 150, 243, 256, 375, 625, 1200, 2187, 3125,
           4096, 4800]


@pytest.mark.parametrize("axis", [0, 1, 2])
@pytest.mark.parametrize("fp32", [False, True])
def test_every_length_on_every_axis(fh, axis, fp32):
    rng = np.random.default_rng(11 + axis)
    for m in LENGTHS:
        shape, padded = [2, 3, 3], [3, 5, 5]
        shape[axis], padded[axis] = (m + 1) // 2, m
        q = rng.standard_normal((3,) + tuple(shape))
        got = fh.grid_convolution(q, padded, 1e-3, fp32=fp32)
        want = reference(q, padded, 1e-3)
        err = np.max(np.abs(got - want)) / np.max(np.abs(want))
        assert err < (4e-6 if fp32 else 1e-12), (m, axis, fp32, err)


@pytest.mark.parametrize("n,m", [((5, 17, 9), (9, 36, 18)), ((130, 3, 11), (270, 5, 24)), ((9, 257, 1), (18, 540, 1)),
                                 ((1, 40, 300), (1, 80, 600))])
@pytest.mark.parametrize("fp32", [False, True])
def test_tail_tiles_and_wider_padding(fh, n, m, fp32):
    rng = np.random.default_rng(3)
    q = rng.standard_normal((2,) + n)
    got = fh.grid_convolution(q, m, 2e-5, fp32=fp32)
    want = reference(q, m, 2e-5)
    err = np.max(np.abs(got - want)) / np.max(np.abs(want))
    assert err < (4e-6 if fp32 else 1e-12), err
