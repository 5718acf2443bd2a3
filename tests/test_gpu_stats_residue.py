"""GPU: norms behind very large samples and on large offsets, and the
correlations reported with them.

The statistics' sums of squares run on from window to window for 64 windows: a
spike of S standard deviations must leave nothing of its S^2 in the windows
behind it, and the rounding of an offset's mean nothing in any.  Exact values in
rational arithmetic; the reported correlation is held to the error bound that
the call states (and 1e-15 for the check's own rounding).
"""
import math
from fractions import Fraction

import numpy as np
import pytest

from test_gpu_stats import check

pytestmark = pytest.mark.gpu


def spiked(n, size, seed):
    rng = np.random.default_rng(seed)
    x = rng.standard_normal(n)
    x[rng.choice(n, 6, replace=False)] = size * rng.choice([-1.0, 1.0], 6)
    return x


@pytest.mark.parametrize("m", [16, 100, 513])
@pytest.mark.parametrize("size", [1e8, 1e10, 1e12, 1e14, 1e18])
def test_norms_behind_spikes(gpu_engine, size, m):
    check(gpu_engine, spiked(2100, size, 5), m)


@pytest.mark.parametrize("offset,spread", [(1e9, 1.0), (1e9, 1e-2), (-1e12, 1.0)])
def test_norms_on_offsets(gpu_engine, offset, spread):
    check(gpu_engine, offset + spread * np.random.default_rng(6).standard_normal(2100), 100)


@pytest.mark.parametrize("precision", ["double", "mixed"])
@pytest.mark.parametrize("size", [1e10, 1e12, 1e16])
def test_reported_correlation(gpu_engine, size, precision):
    n, m = 1500, 40
    x = spiked(n, size, 7)
    r = gpu_engine.join(x, None, m, precision=precision, return_corr=True)
    _, idx = gpu_engine.unpack_profile(r["profile_a"])
    q = [Fraction(v) for v in x.tolist()]
    total = [sum(q[w:w + m]) for w in range(n - m + 1)]
    ssd = [float(sum(v * v for v in q[w:w + m]) - total[w] ** 2 / m) for w in range(n - m + 1)]
    assert (idx >= 0).all()
    for w, j in enumerate(idx.tolist()):
        dot = sum(a * b for a, b in zip(q[w:w + m], q[j:j + m])) - total[w] * total[j] / m
        want = float(dot) / math.sqrt(ssd[w] * ssd[j])
        assert abs(r["corr_a"][w] - want) <= r["max_abs_r_err"] + 1e-15, (w, j)
