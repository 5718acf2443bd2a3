"""GPU: seeds of the FP64 band kernel beside a large sample.

A thread's four diagonals share a centre for their seeds unless the windows'
means lie too far apart.  Here a spike leaves with the first of them: B repeats
A's samples after the spike, so on one diagonal every correlation is 1, the only
ones above the threshold, and the sums show the error of that diagonal's seed.
Four places of the spike put the diagonal at each place in its thread.  1e-11
leaves room for the recurrence's rounding over the rows of a segment (3000 x
2^-53); a seed centred 1e12 / 64 away is off by some 1e-7.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("p", [200, 201, 202, 203])
def test_spike_leaves_with_the_first_window(gpu_engine, p):
    m, nb = 64, 3000
    a = np.random.default_rng(9).standard_normal(p + 1 + nb)
    b = a[p + 1:].copy()
    a[p] = 1e12
    r = gpu_engine.join(a, b, m, "SUM_THRESH", "double", threshold=0.99, keep_rows=True)
    assert np.max(np.abs(r["sum_b"] - 1.0)) <= 1e-11
    assert np.max(np.abs(r["sum_a"][p + 1:] - 1.0)) <= 1e-11
