"""GPU: matrix summaries whose entries' largest correlations are negative.

With a threshold below 0 a grid entry of anti-correlated windows (a rising
stretch against a falling one) has a negative maximum, which has to be
reported, and the band kernel's blocks past the last window count nowhere.
Amplitudes of 1, 100 and 1e-3 move the windows' norms to both sides of 1.
Both forms, against brute-force correlation matrices; the mixed form's
tolerance is its own.
"""
import numpy as np
import pytest

from parity import TOL_MIXED
from test_gpu_experimental import TOL, check_matrix, corr_matrix
from test_gpu_exact_lists import self_matrix

pytestmark = pytest.mark.gpu


def ramps(n, scale, seed):
    """Rising, then falling, with noise."""
    x = np.minimum(np.arange(n), np.arange(n)[::-1]) / 20.0
    return scale * (x + 0.3 * np.random.default_rng(seed).standard_normal(n))


@pytest.mark.parametrize("precision", ["double", "mixed"])
@pytest.mark.parametrize("thr", [-1.0, -0.99, -0.2])
@pytest.mark.parametrize("scale", [1.0, 100.0, 1e-3])
@pytest.mark.parametrize("n,nb,m,h,w", [(4099, None, 100, 4, 4), (3000, 1100, 50, 5, 40),
                                        (2210, 3100, 400, 13, 9)])
def test_negative_entries(gpu_engine, precision, thr, scale, n, nb, m, h, w):
    a = ramps(n, scale, 1)
    b = None if nb is None else ramps(nb, scale, 2)
    r = gpu_engine.join(a, b, m, "MATRIX_SUMMARY", precision, threshold=thr, matrix_height=h,
                        matrix_width=w)
    assert r["counters"]["steps"] > 0  # the band kernel, not the visit kernel
    if b is None:
        C = self_matrix(a, m)
        i = np.arange(len(C))
        C[i[:, None] > i[None, :]] = np.nan  # a self-join walks the upper triangle
    else:
        C = corr_matrix(b, a, m)
    check_matrix(r["matrix"].astype(np.float64), C, h, w, thr,
                 TOL if precision == "double" else TOL_MIXED)
