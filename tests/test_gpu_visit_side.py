"""GPU: k-best lists and matrix summaries against the FP64 visit kernels.

Double and mixed joins of these types run the band kernel; ULTRA still walks every
cell in FP64 (the visit kernels), so it is the side that shares none of their
code.  Values agree within float32 rounding (double) or the mixed form's
tolerance; entries present on one side only lie at the threshold's edge.
"""
import numpy as np
import pytest

from parity import TOL_MIXED
from test_gpu_experimental import TOL

pytestmark = pytest.mark.gpu


def series(n, seed):
    x = np.cumsum(np.random.default_rng(seed).standard_normal(n))
    x[n // 6:n // 6 + 30] = np.nan
    return x


def agree(got, want, thr, tol):
    both = (got >= -1) & (want >= -1)
    assert both.any()
    assert np.max(np.abs(got[both] - want[both])) <= tol
    only = (got >= -1) != (want >= -1)
    assert np.all(np.abs(np.maximum(got, want)[only] - thr) <= tol)


@pytest.mark.parametrize("precision,tol", [("double", TOL), ("mixed", TOL_MIXED)])
@pytest.mark.parametrize("nb", [None, 9001])
@pytest.mark.parametrize("k", [1, 5])
def test_lists(gpu_engine, precision, tol, nb, k):
    a, b, m, thr = series(12000, 1), None if nb is None else series(nb, 2), 128, 0.6
    kw = dict(threshold=thr, max_matches=k, keep_rows=nb is not None)
    want = gpu_engine.join(a, b, m, "ALL_NEIGHBORS", "ultra", **kw)
    got = gpu_engine.join(a, b, m, "ALL_NEIGHBORS", precision, **kw)
    assert got["counters"]["steps"] > 0 and want["counters"]["steps"] == 0
    for side in ("knn_a",) if nb is None else ("knn_a", "knn_b"):
        cw, cg = (gpu_engine.unpack_profile(r[side])[0].astype(np.float64) for r in (want, got))
        agree(cg, cw, thr, tol)


@pytest.mark.parametrize("precision,tol", [("double", TOL), ("mixed", TOL_MIXED)])
@pytest.mark.parametrize("nb", [None, 9001])
@pytest.mark.parametrize("thr", [0.5, -0.9])
def test_grids(gpu_engine, precision, tol, nb, thr):
    a, b = series(12000, 3), None if nb is None else series(nb, 4)
    kw = dict(threshold=thr, matrix_height=40, matrix_width=31)
    want = gpu_engine.join(a, b, 100, "MATRIX_SUMMARY", "ultra", **kw)
    got = gpu_engine.join(a, b, 100, "MATRIX_SUMMARY", precision, **kw)
    assert got["counters"]["steps"] > 0 and want["counters"]["steps"] == 0
    agree(got["matrix"].astype(np.float64), want["matrix"].astype(np.float64), thr, tol)


@pytest.mark.parametrize("k", [16, 17])
def test_either_side_of_the_list_line(gpu_engine, k):
    """Lists of more than 16 from long windows of a short series go to the visit
    kernel itself; the values are the same on both sides of the line."""
    a, m, thr = series(12000, 5), 600, 0.4
    kw = dict(threshold=thr, max_matches=k)
    want = gpu_engine.join(a, None, m, "ALL_NEIGHBORS", "ultra", **kw)
    got = gpu_engine.join(a, None, m, "ALL_NEIGHBORS", "double", **kw)
    assert (got["counters"]["steps"] > 0) == (k == 16)
    cw, cg = (gpu_engine.unpack_profile(r["knn_a"])[0].astype(np.float64) for r in (want, got))
    agree(cg, cw, thr, TOL)
