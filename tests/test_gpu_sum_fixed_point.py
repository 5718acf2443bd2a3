"""GPU: double-precision SUM_THRESH, whose slab sums are fixed point.

Negative thresholds (terms of both signs), correlations of 1 up to rounding
(exact repeats, the largest terms), and sizes at the edges of the FP64 band
kernel's 512-diagonal bands, 64-row slabs and segments.  A sum's terms are cut
at 2^-53, so it differs from the oracle's FP64 sum by rounding: 1e-9 relative
covers both, far below one term.
"""
import numpy as np
import pytest

from parity import check_sum

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind,thr", [("walk", -1.0), ("walk", -0.3), ("walk", 0.0),
                                      ("repeats", 0.999), ("gaps", 0.6)])
@pytest.mark.parametrize("n,nb,m", [(70, None, 5), (600, None, 24), (1024 + 63, 577, 64),
                                    (4600, None, 333)])
def test_sums(gpu_engine, oracle_mod, kind, thr, n, nb, m):
    rng = np.random.default_rng(n + m)

    def series(k):
        x = np.cumsum(rng.standard_normal(k))
        if kind == "repeats":
            x = np.tile(rng.standard_normal(2 * m + 1), k // (2 * m + 1) + 1)[:k]
        elif kind == "gaps":
            x[rng.choice(k, 3, replace=False)] = np.nan
        return x

    a = series(n)
    b = None if nb is None else series(nb)
    got = gpu_engine.join(a, b, m, "SUM_THRESH", "double", threshold=thr, keep_rows=nb is not None)
    want = oracle_mod.join(a, b, m, "SUM_THRESH", threshold=thr, keep_rows=nb is not None,
                           exact_flat=True)
    check_sum(kind + "/A", got["sum_a"], want["sum_a"], thr, 1e-9)
    if nb is not None:
        check_sum(kind + "/B", got["sum_b"], want["sum_b"], thr, 1e-9)
