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


@pytest.mark.parametrize("kind,n,seed,m,named", [
    ("sine", 9000, 3, 64, {84: 2030, 289: 6127, 341: 1314, 342: 1315, 531: 5396, 820: 5685,
                           823: 5688, 1172: 3118}),
    ("spikes", 20000, 1, 100, {13622: 16490, 13624: 7654, 16504: 11736, 18180: 13610})])
def test_without_seeds(gpu_engine, kind, n, seed, m, named):
    rng = np.random.default_rng(seed)
    if kind == "sine":
        x = np.sin(np.arange(n) * 2 * np.pi / 97.3) + .001 * rng.standard_normal(n)
    else:
        x = rng.standard_normal(n)
        x[rng.choice(n, n // 2000 + 1, replace=False)] += 1e4
    got = partners(gpu_engine, x, m)
    assert {w: int(got[w]) for w in named} == named
