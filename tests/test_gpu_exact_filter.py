"""GPU: double-precision 1NN joins large enough for the FP32 filter.

The filter may only skip cells that its error bound rules out, so the profile
has to be the FP64 one on every kind of series, also where FP32 carries
little (spikes, large offsets, near-flat windows), where it cannot be used
(magnitudes out of its range: the FP64 band kernel runs) and where it rules
out nothing (exact repeats).  Sizes sit at the edges of its 1024-diagonal
bands, 128-row slabs and 512-sample anchor passes.
"""
import numpy as np
import pytest

from parity import TOL_FP64, check_1nn_direct

pytestmark = pytest.mark.gpu


def series(kind, n, seed):
    rng = np.random.default_rng(seed)
    x = np.cumsum(rng.standard_normal(n))
    if kind == "noise":
        x = rng.standard_normal(n)
    elif kind == "spikes":
        x = rng.standard_normal(n)
        x[rng.choice(n, 6, replace=False)] += 1e6
    elif kind == "gaps":
        x[rng.choice(n, 12, replace=False)] = np.nan
        x[n // 2:n // 2 + 300] = np.inf
    elif kind == "nearflat":
        for _ in range(6):
            p = int(rng.integers(0, n - 600))
            x[p:p + 500] = x[p] + 1e-4 * rng.standard_normal(500)
    elif kind == "offset":
        x = 1e9 + 1e-2 * x
    elif kind == "huge":
        x = 1e20 * x
    elif kind == "repeats":
        x = np.tile(np.round(4 * rng.standard_normal(160)), n // 160 + 1)[:n]
    return x


@pytest.mark.parametrize("kind", ["walk", "noise", "spikes", "gaps", "nearflat", "offset", "huge",
                                  "repeats"])
@pytest.mark.parametrize("n,nb,m", [(9001, None, 64), (1024 * 9 + 95, None, 96), (7000, 6007, 513)])
def test_double_profile(gpu_engine, oracle_mod, kind, n, nb, m):
    a = series(kind, n, 1)
    b = None if nb is None else series(kind, nb, 2)
    got = gpu_engine.join(a, b, m, precision="double", keep_rows=nb is not None, return_corr=True)
    want = oracle_mod.join(a, b, m, "1NN_INDEX", keep_rows=nb is not None, exact_flat=True)
    if kind == "huge":
        assert got["counters"]["verifications"] == 0
    else:
        assert got["counters"]["verifications"] > 0
    other = a if b is None else b
    _, gi = gpu_engine.unpack_profile(got["profile_a"])
    check_1nn_direct(kind + "/A", got["corr_a"], gi, want["idx_a"], TOL_FP64, a, other, m)
    if nb is not None:
        _, gi = gpu_engine.unpack_profile(got["profile_b"])
        check_1nn_direct(kind + "/B", got["corr_b"], gi, want["idx_b"], TOL_FP64, b, a, m)


@pytest.mark.parametrize("n,m", [(12000, 700), (9000, 1500)])
def test_more_requests_than_worth_verifying(gpu_engine, oracle_mod, n, m):
    """Exact repeats of every window: the join's limit of requests leaves
    units to the FP64 band kernel midway, whose requests must be void."""
    a = (np.arange(n) // 25 % 2).astype(float)
    got = gpu_engine.join(a, None, m, precision="double", return_corr=True)
    want = oracle_mod.join(a, None, m, "1NN_INDEX", exact_flat=True)
    _, gi = gpu_engine.unpack_profile(got["profile_a"])
    check_1nn_direct("square", got["corr_a"], gi, want["idx_a"], TOL_FP64, a, a, m)
