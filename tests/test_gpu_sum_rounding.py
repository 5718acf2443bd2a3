"""GPU: terms of double-precision sums are rounded to the sums' unit, not cut.

On integers of window 64 the means, covariances and their recurrence are exact
dyadic fractions, so every cell's FP64 correlation is known to the last bit from
the engine's own inverse norms, and the sums of those above 0 can be formed
exactly.  A sum's terms are kept in units of 2^-53: cut, a term between 1/4 and 1/2
loses 2^-55 on average and smaller ones up to 2^-53, about 0.8 x 2^-54 here.  The
rest of a sum's error, the rounding of its few dozen FP64 additions (2^-45 at most
each), has no sign, so over 4097 windows the mean error stays below 0.2 x 2^-54
per term.
"""
import math

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_terms_are_rounded(gpu_engine):
    m, ns = 64, 4097
    x = np.random.default_rng(8).integers(-8, 9, ns + m - 1).astype(np.float64)
    got = gpu_engine.join(x, None, m, "SUM_THRESH", "double", threshold=0.0)["sum_a"]
    _, inv, _, _ = gpu_engine.window_stats(x, m)
    w = np.lib.stride_tricks.sliding_window_view(x, m)
    w = w - w.mean(axis=1, keepdims=True)
    i, j = np.indices((ns, ns), sparse=True)
    # the cell (i, j), i < j, is (cov inv_j) inv_i
    r = (w @ w.T) * inv[None, :] * inv[:, None]
    r = np.where(i < j, r, r.T)
    r[(np.abs(i - j) < m // 4) | ~(r > 0)] = 0.0
    assert 1000 < np.count_nonzero(r[0]) < 3000 and r.max() < 1
    error = np.array([got[k] - math.fsum(r[k]) for k in range(ns)])
    assert np.max(np.abs(error)) <= 64 * 2.0 ** -45 + np.count_nonzero(r, axis=1).max() * 2.0 ** -54
    assert abs(error.mean()) <= 0.2 * 2.0 ** -54 * np.count_nonzero(r) / ns
