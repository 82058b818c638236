"""The grid convolution of thin grids (4 to 16 points along axis 2: two
transformed axes and the product along the third) at the ends of that range
and of the shared memory, with one, two and three transform stages per axis
and an odd number of fields, against numpy's FFT.

Tolerances: those of a transform over three axes, 2 u log2(P) in the 2-norm
times a small factor to the max-norm (4e-6 in FP32, 1e-12 in FP64); the
product's sums of up to 16 terms add less than one more transform stage."""
import numpy as np
import pytest

from test_gpu_fftconv import reference

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n2,m2", [(3, 5), (4, 8), (5, 9), (7, 15), (8, 15), (9, 18), (12, 24), (15, 30), (16, 32),
                                   (17, 36)])
@pytest.mark.parametrize("n0,m0,n1,m1", [(1, 1, 1, 1), (3, 6, 8, 16), (2, 5, 61, 125), (40, 90, 7, 15),
                                         (33, 75, 70, 150), (601, 1215, 2, 4), (2, 3, 1300, 2700)])
@pytest.mark.parametrize("fp32", [False, True])
def test_thin_grids(fh, n0, m0, n1, m1, n2, m2, fp32):
    rng = np.random.default_rng(n0 + 10 * n1 + 100 * n2)
    q = rng.standard_normal((3, n0, n1, n2))
    got = fh.grid_convolution(q, (m0, m1, m2), 1e-3, fp32=fp32)
    want = reference(q, (m0, m1, m2), 1e-3)
    err = np.max(np.abs(got - want)) / np.max(np.abs(want))
    assert err < (4e-6 if fp32 else 1e-12), err
