"""GPU: double-precision k-best lists and matrix summaries large enough for
the FP32 filter, against brute-force correlation matrices.

The filter may only skip cells that its bounds rule out, so lists and grids
must be the FP64 ones.  Lists take it at every size, grids from entries of
64 windows on; sizes sit at that edge, at the edges of its 1024-diagonal
bands, and where a window has fewer bands or cells than its list entries.  Tolerance as in the brute-force checks it reuses:
float32 rounding of an FP64 correlation.
"""
import numpy as np
import pytest

from test_gpu_experimental import check_knn, check_matrix, corr_matrix

pytestmark = pytest.mark.gpu


def series(kind, n, seed):
    rng = np.random.default_rng(seed)
    x = np.cumsum(rng.standard_normal(n))
    if kind == "gaps":
        x[rng.choice(n, 5, replace=False)] = np.nan
        x[n // 3:n // 3 + 90] = np.inf
    elif kind == "spikes":
        x = rng.standard_normal(n)
        x[rng.choice(n, 3, replace=False)] += 1e6
    return x


def self_matrix(a, m):
    C = corr_matrix(a, a, m)
    i = np.arange(len(C))
    C[np.abs(i[:, None] - i[None, :]) < m // 4] = np.nan
    return C


@pytest.mark.parametrize("kind", ["walk", "gaps", "spikes"])
@pytest.mark.parametrize("n,nb,m,k,thr", [(2048 + 31, None, 32, 1, 0.3), (4200, None, 50, 2, -0.2),
                                          (2300, 2048 + 49, 50, 1, 0.5)])
def test_lists(gpu_engine, kind, n, nb, m, k, thr):
    a = series(kind, n, 1)
    b = None if nb is None else series(kind, nb, 2)
    r = gpu_engine.join(a, b, m, "ALL_NEIGHBORS", "double", threshold=thr, max_matches=k,
                        keep_rows=nb is not None)
    assert r["counters"]["steps"] > 0  # the filter ran
    C = self_matrix(a, m) if b is None else corr_matrix(b, a, m)
    check_knn(gpu_engine, r["knn_a"], k, C, thr, kind + "/A")
    if b is not None:
        check_knn(gpu_engine, r["knn_b"], k, C.T, thr, kind + "/B")


@pytest.mark.parametrize("kind", ["walk", "gaps", "spikes", "square"])
@pytest.mark.parametrize("n,nb,m,k,thr", [(300, None, 16, 64, 0.0), (1100, 330, 30, 7, 0.2),
                                          (1023 + 32, None, 32, 64, -1.0), (2600, None, 50, 20, 0.4)])
def test_short_lists(gpu_engine, kind, n, nb, m, k, thr):
    """Fewer bands than list entries, lists longer than a window has cells,
    exact repeats (no bound separates their cells)."""
    def make(length, seed):
        if kind == "square":
            return (np.arange(length) // 7 % 2).astype(float)
        return series(kind, length, seed)

    a = make(n, 4)
    b = None if nb is None else make(nb, 5)
    r = gpu_engine.join(a, b, m, "ALL_NEIGHBORS", "double", threshold=thr, max_matches=k,
                        keep_rows=nb is not None)
    assert r["counters"]["steps"] > 0
    C = self_matrix(a, m) if b is None else corr_matrix(b, a, m)
    check_knn(gpu_engine, r["knn_a"], k, C, thr, kind + "/A")
    if b is not None:
        check_knn(gpu_engine, r["knn_b"], k, C.T, thr, kind + "/B")


def test_lists_merge_given_entries(gpu_engine):
    """Given entries keep their places: one above every match, one below."""
    n, m, k = 4200, 40, 2
    a = series("walk", n, 3)
    ns = n - m + 1
    none = gpu_engine.join(a, None, m, "ALL_NEIGHBORS", "double", threshold=0.5, max_matches=k)
    given = np.full(ns * k, gpu_engine.NO_MATCH, dtype=np.uint64)
    top = np.uint64(int(np.float32(1.0).view(np.uint32)) | (7 << 32))
    given[0::2 * k] = top          # every other window: a best of 1
    r = gpu_engine.join(a, None, m, "ALL_NEIGHBORS", "double", threshold=0.5, max_matches=k,
                        profile_a=given)
    want, got = none["knn_a"].reshape(ns, k), r["knn_a"].reshape(ns, k)
    assert np.array_equal(got[1::2], want[1::2])
    assert np.all(got[0::2, 0] == top)
    assert np.array_equal(got[0::2, 1], want[0::2, 0])


@pytest.mark.parametrize("kind", ["walk", "gaps", "spikes"])
@pytest.mark.parametrize("n,nb,m,h,w,thr", [(2085, None, 32, 32, 32, 0.0), (3100, None, 65, 7, 41, 0.4),
                                            (3000, 1100, 50, 5, 40, -0.3)])
def test_grids(gpu_engine, kind, n, nb, m, h, w, thr):
    a = series(kind, n, 4)
    b = None if nb is None else series(kind, nb, 5)
    r = gpu_engine.join(a, b, m, "MATRIX_SUMMARY", "double", threshold=thr, matrix_height=h,
                        matrix_width=w)
    assert r["counters"]["steps"] > 0  # the filter ran
    if b is None:
        C = self_matrix(a, m)
        i = np.arange(len(C))
        C[i[:, None] > i[None, :]] = np.nan  # a self-join walks the upper triangle
    else:
        C = corr_matrix(b, a, m)
    check_matrix(r["matrix"], C, h, w, thr)
