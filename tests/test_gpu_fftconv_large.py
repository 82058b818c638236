"""The grid convolution on a torus of more than 2^31 points, whose last places
along axis 0 lie beyond 32-bit indices, against the direct sum over a few
sources.

Tolerances: 2 u log2(P) in the 2-norm (P = 2.2e9: 3.8e-6 in FP32, 7e-15 in
FP64) and a factor of two from the potentials' 2-norm per point to their
largest."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("fp32", [False, True])
def test_more_points_than_32_bits_count(fh, fp32):
    n, m, h = (3, 2, 40), (4800, 4800, 96), 1e-3
    assert m[0] * m[1] * m[2] > 2 ** 31
    q = np.random.default_rng(8).standard_normal((2,) + n)
    try:
        got = fh.grid_convolution(q, m, h, fp32=fp32)
    finally:
        fh.release_cached_memory()
    at = np.stack(np.meshgrid(*[np.arange(k) for k in n], indexing="ij"), axis=-1).reshape(-1, 3)
    d = np.sqrt((((at[:, None] - at[None]) ** 2).sum(-1)).astype(float))
    kernel = np.where(d > 0, 1.0 / (h * np.where(d > 0, d, 1.0)), 0.0)
    want = (q.reshape(2, -1) @ kernel).reshape(q.shape)
    err = np.max(np.abs(got - want)) / np.max(np.abs(want))
    assert err < (8e-6 if fp32 else 1.4e-14), err
