"""GPU: mixed 1NN joins keep their partners where FP32 leaves several.

Cells whose correlations lie about 1e-6 apart may have equal FP32 values; the
one that the join publishes first is then the reported partner, so the order
of the band kernel's exact path shows in the profile.  The partners here are
those of the row-by-row exact path (and, in joins without seeds, of filters
that start from nothing).
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def partners(gpu_engine, a, m):
    return gpu_engine.unpack_profile(gpu_engine.join(a, None, m, precision="mixed")["profile_a"])[1]


def test_long_windows(gpu_engine):
    # two cells of one column, in neighbouring warps: rows 734017 (distance
    # 6.08349) and 734018 (6.08367).  Warps may overtake each other, hence
    # nine of ten joins.
    rng = np.random.default_rng(115)
    n = 1 << 20
    x = np.cumsum(rng.standard_normal(n))
    x = x + 0.5 * rng.standard_normal(n)
    named = [int(partners(gpu_engine, x, 1024)[780609]) for _ in range(10)]
    assert named.count(734017) >= 9, named
