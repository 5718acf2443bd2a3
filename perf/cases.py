"""Workloads that stand for what users of the matrix-profile engine run.

Every case is one call (or one call and the unpacking of its packed result)
through the public Python front of the engine.  The listed cases follow the
reference's own interfaces: pyscamp's functions default to double precision,
so most of them do, and the mixed form is what the long joins use.

``kind`` is the entry point, ``data`` the distribution of the series:
  walk   random walk (the benchmarks' base series)
  noisy  random walk plus white noise (the 2^24-sample benchmark)
  motif  random walk with planted noisy sinusoids and 0.1% NaN samples
         (the AB benchmark)
  gaps   random walk with 1% of its samples in NaN gaps
  beat   a sinusoid of slowly varying period plus white noise: a machine or
         heart-beat recording, whose windows all have many close matches
"""
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.getcwd(), "gpu-scrimp-large_gb300"))

import scamp_gb300  # noqa: E402

# Floating operations of one cell of the distance matrix: two fused
# multiply-adds along its diagonal, two multiplications by the inverse norms.
_CELL_FLOPS = 6


def listed():
    return [
        # the smallest call: a notebook's or a unit test's series
        {"name": "self_1k", "kind": "selfjoin", "n": 1000, "m": 50, "precision": "double",
         "data": "walk"},
        # an ordinary recording: a day of minutes, a few minutes of a sensor
        {"name": "self_10k_beat", "kind": "selfjoin", "n": 10007, "m": 100,
         "precision": "double", "data": "beat"},
        # the reference's self-join benchmark (131072 samples, m = 100)
        {"name": "self_128k", "kind": "selfjoin", "n": 131072, "m": 100, "precision": "double",
         "data": "walk"},
        # long windows over a recording with drop-outs
        {"name": "self_40k_gaps_m1024", "kind": "selfjoin", "n": 40009, "m": 1024,
         "precision": "double", "data": "gaps"},
        # one recording searched in another (the AB benchmark, scaled down)
        {"name": "ab_60k_30k_m256", "kind": "abjoin", "n": 60000, "nb": 30011, "m": 256,
         "precision": "double", "data": "motif"},
        # the long self-join the mixed form is for (the 2^24-sample benchmark's
        # series and window, at a sixteenth of its length)
        {"name": "self_1m_mixed_m1024", "kind": "selfjoin", "n": 1 << 20, "m": 1024,
         "precision": "mixed", "data": "noisy"},
        # device-resident AB join keeping both profiles, mixed: one step of a
        # pipeline whose series are already on the GPU
        {"name": "ab_device_256k_128k_mixed", "kind": "abdevice", "n": 1 << 18,
         "nb": (1 << 17) + 5, "m": 256, "precision": "mixed", "data": "motif"},
        # how often each pattern repeats: sums of correlations over a threshold
        {"name": "sum_32k", "kind": "sum", "n": 32768, "m": 128, "precision": "double",
         "data": "walk", "threshold": 0.9},
        {"name": "sum_200k_mixed", "kind": "sum", "n": 200003, "m": 256, "precision": "mixed",
         "data": "noisy", "threshold": 0.5},
        # the five best matches of every window
        {"name": "knn_20k", "kind": "knn", "n": 20011, "m": 128, "precision": "double",
         "data": "walk", "threshold": 0.5, "k": 5},
        # a picture of the whole distance matrix
        {"name": "matrix_30k", "kind": "matrix", "n": 30000, "m": 100, "precision": "double",
         "data": "noisy", "threshold": 0.0, "side": 50},
        # many short series in one call (the batch benchmark's lengths and
        # windows, a sixteenth of its count)
        {"name": "batch_256", "kind": "batch", "n": 256, "lo": 10, "hi": 14,
         "precision": "mixed", "data": "walk"},
    ]


def _log_int(rng, lo, hi):
    return int(round(lo * (hi / lo) ** rng.random()))


def draw(rng):
    kind = rng.choice(["selfjoin", "selfjoin", "selfjoin", "abjoin", "abdevice", "sum", "knn",
                       "matrix", "batch"])
    if kind == "batch":
        lo = rng.uniform(10.0, 12.0)
        return {"kind": kind, "n": _log_int(rng, 32, 256), "lo": round(lo, 3),
                "hi": round(lo + rng.uniform(0.5, 2.0), 3), "precision": "mixed", "data": "walk"}
    data = rng.choice(["walk", "noisy", "motif", "gaps", "beat"])
    precision = "mixed" if kind == "abdevice" else rng.choice(["double", "double", "mixed"])
    if kind == "selfjoin":
        n = _log_int(rng, 1000, 131072 if precision == "double" else 1 << 19)
    elif kind == "abjoin":
        n = _log_int(rng, 1000, 90000 if precision == "double" else 1 << 19)
    elif kind == "abdevice":
        n = _log_int(rng, 4000, 1 << 18)
    elif kind == "sum":
        n = _log_int(rng, 2000, 40000 if precision == "double" else 200003)
    else:
        n = _log_int(rng, 2000, 32000)
    m = _log_int(rng, 32, min(1024, n // 16))
    case = {"kind": kind, "n": n, "m": m, "precision": precision, "data": data}
    if kind in ("abjoin", "abdevice"):
        case["nb"] = max(2 * m, _log_int(rng, max(n // 8, 500), n))
    if kind == "sum":
        case["threshold"] = round(rng.uniform(0.5, 0.95), 3)
    if kind == "knn":
        case["threshold"] = round(rng.uniform(0.3, 0.8), 3)
        case["k"] = rng.randint(1, 10)
    if kind == "matrix":
        case["threshold"] = 0.0
        case["side"] = rng.randint(20, 100)
    return case


# --------------------------------------------------------------------------
# Series
# --------------------------------------------------------------------------
def _series(rng, n, m, data):
    if data == "beat":
        period = 80.0 * (1.0 + 0.05 * np.cumsum(rng.standard_normal(n)) / np.sqrt(n))
        return np.sin(2 * np.pi * np.cumsum(1.0 / period)) + 0.1 * rng.standard_normal(n)
    x = np.cumsum(rng.standard_normal(n))
    if data == "noisy":
        x = x + 0.5 * rng.standard_normal(n)
    elif data == "gaps":
        covered = 0
        while covered < n // 100:
            length = int(rng.integers(1, max(2, min(500, n // 100))))
            p = int(rng.integers(0, n - length))
            x[p:p + length] = np.nan
            covered += length
    elif data == "motif":
        length = min(256, n // 32)
        shapes = np.random.default_rng(1000)
        for p in rng.choice(n // length, size=max(1, n // length // 16), replace=False) * length:
            t = np.arange(length)
            x[p:p + length] = (np.sin(2 * np.pi * t / shapes.uniform(20, 200)) +
                               0.1 * rng.standard_normal(length))
        x[rng.choice(n, size=n // 1000, replace=False)] = np.nan
    return x


def _batch(case, rng):
    # the lengths and windows belong to the case, the samples to the seed
    shape = np.random.default_rng(case["n"])
    out, windows = [], []
    for _ in range(case["n"]):
        n = int(round(2 ** shape.uniform(case["lo"], case["hi"])))
        windows.append(int(shape.choice([32, 64, 128])))
        x = np.cumsum(rng.standard_normal(n))
        out.append(x * 10 ** rng.uniform(-3, 3) + rng.uniform(-1e4, 1e4))
    return out, windows


def _inputs(case, seed):
    rng = np.random.default_rng(seed)
    if case["kind"] == "batch":
        return _batch(case, rng)
    a = _series(rng, case["n"], case["m"], case["data"])
    b = _series(rng, case["nb"], case["m"], case["data"]) if "nb" in case else None
    return a, b


def prepare(case, seed):
    a, b = _inputs(case, seed)
    state = {"case": case, "a": a, "b": b}
    if case["kind"] == "abdevice":
        # a pipeline's resident series and profile buffers
        dev = torch.device("cuda")
        m = case["m"]
        state["a"], state["b"] = torch.from_numpy(a).to(dev), torch.from_numpy(b).to(dev)
        state["pa"] = torch.empty(len(a) - m + 1, dtype=torch.int64, device=dev)
        state["pb"] = torch.empty(len(b) - m + 1, dtype=torch.int64, device=dev)
        state["ca"] = torch.empty(len(a) - m + 1, dtype=torch.float64, device=dev)
        state["cb"] = torch.empty(len(b) - m + 1, dtype=torch.float64, device=dev)
    return state


# an empty entry of a packed profile, as a signed integer
_NO_MATCH = int(scamp_gb300.NO_MATCH.astype(np.int64))


def run(state):
    case, a, b = state["case"], state["a"], state["b"]
    kind, precision = case["kind"], case["precision"]
    if kind == "selfjoin":
        return scamp_gb300.selfjoin(a, case["m"], precision=precision)
    if kind == "abjoin":
        return scamp_gb300.abjoin(a, b, case["m"], precision=precision)
    if kind == "abdevice":
        pa, pb, ca, cb = state["pa"], state["pb"], state["ca"], state["cb"]
        pa.fill_(_NO_MATCH)
        pb.fill_(_NO_MATCH)
        scamp_gb300.join_device(
            a.data_ptr(), a.numel(), case["m"], b.data_ptr(), b.numel(), precision=precision,
            keep_rows=True, profile_a_ptr=pa.data_ptr(), profile_b_ptr=pb.data_ptr(),
            corr_a_ptr=ca.data_ptr(), corr_b_ptr=cb.data_ptr(),
            stream=torch.cuda.current_stream().cuda_stream)
        return ca, pa >> 32, cb, pb >> 32
    if kind == "sum":
        return scamp_gb300.selfjoin_sum(a, case["m"], precision=precision,
                                        threshold=case["threshold"])
    if kind == "knn":
        r = scamp_gb300.join(a, None, case["m"], "ALL_NEIGHBORS", precision,
                             threshold=case["threshold"], max_matches=case["k"])
        return scamp_gb300.unpack_profile(r["knn_a"])
    if kind == "matrix":
        return scamp_gb300.selfjoin_matrix(a, case["m"], precision=precision,
                                           threshold=case["threshold"], mheight=case["side"],
                                           mwidth=case["side"])
    # batch: the user's answer is every series' profile
    res = scamp_gb300.join_batch(a, b, precision)
    corr, idx = scamp_gb300.unpack_profile(np.concatenate([r["profile_a"] for r in res]))
    return corr, idx


# --------------------------------------------------------------------------
# Work and exact values
# --------------------------------------------------------------------------
def _cells(case):
    m = case["m"]
    if "nb" in case:
        return float(case["n"] - m + 1) * float(case["nb"] - m + 1)
    k = case["n"] - m + 1 - m // 4  # diagonals from the exclusion zone out
    return 0.5 * k * (k + 1)


def work(case):
    if case["kind"] == "batch":
        # lengths round(2^U[lo, hi]): mean length and mean square over 2
        lo, hi = case["lo"] * np.log(2), case["hi"] * np.log(2)
        n1 = (np.exp(hi) - np.exp(lo)) / (hi - lo)
        n2 = (np.exp(2 * hi) - np.exp(2 * lo)) / (2 * (hi - lo))
        return {"bytes": float(16 * case["n"] * n1),
                "flops": float(_CELL_FLOPS * case["n"] * n2 / 2)}
    samples = case["n"] + case.get("nb", 0)
    windows = case["n"] - case["m"] + 1
    if case["kind"] == "abdevice":
        windows += case["nb"] - case["m"] + 1
    out = {"knn": 8 * case.get("k", 1), "abdevice": 16}.get(case["kind"], 8) * windows
    if case["kind"] == "matrix":
        out = 4 * case["side"] ** 2
    return {"bytes": 8.0 * samples + out, "flops": _CELL_FLOPS * _cells(case)}


def _windows(x, m, dev):
    """Rows of centred windows over their norms (FP64); False where a window
    holds a non-finite sample or has no spread."""
    t = torch.from_numpy(np.array(x)).to(dev)
    bad = ~torch.isfinite(t)
    w = torch.where(bad, torch.zeros_like(t), t).unfold(0, m, 1)
    ok = ~bad.unfold(0, m, 1).any(1)
    w = w - w.mean(1, keepdim=True)
    w = w - w.mean(1, keepdim=True)
    ssd = (w * w).sum(1)
    ok &= ssd > 1e-13
    return w / torch.sqrt(ssd).clamp_min(1e-300)[:, None], ok


def _corr_blocks(za, oka, zb, okb, excl):
    """Blocks of the correlation matrix (rows: windows of a; -3 where a cell
    does not count), as (first row, block)."""
    nb = zb.shape[0]
    step = max(1, min(za.shape[0], (1 << 28) // nb))
    col = torch.arange(nb, device=zb.device)
    for i in range(0, za.shape[0], step):
        r = za[i:i + step] @ zb.T
        r.clamp_(-1.0, 1.0)
        r.masked_fill_(~okb[None, :], -3.0)
        r.masked_fill_(~oka[i:i + step, None], -3.0)
        if excl > 0:
            rows = torch.arange(i, i + r.shape[0], device=zb.device)
            r.masked_fill_((rows[:, None] - col[None, :]).abs() < excl, -3.0)
        yield i, r


def _distance(r, m):
    d = torch.sqrt((2.0 * m * (1.0 - r)).clamp_min(0.0))
    return torch.where(r < -1, torch.full_like(d, float("nan")), d)


def _best(za, oka, zb, okb, excl):
    return torch.cat([r.max(1).values for _, r in _corr_blocks(za, oka, zb, okb, excl)])


def exact(case, seed):
    dev = torch.device("cuda" if torch.cuda.is_available() else "cpu")
    a, b = _inputs(case, seed)
    if case["kind"] == "batch":
        if case["n"] * 2.0 ** (2 * case["hi"]) * 128 > 3e13:
            return None
        out = []
        for x, m in zip(a, b):
            z, ok = _windows(x, m, dev)
            out.append(_best(z, ok, z, ok, m // 4))
        return torch.cat(out).cpu().numpy(), None
    m = case["m"]
    samples_b = case.get("nb", case["n"])
    # the whole matrix by FP64 products: skipped where it takes too long or
    # where the window matrix does not fit
    if 2.0 * case["n"] * samples_b * m > 6e12 or 8.0 * case["n"] * m > 3e10:
        return None
    za, oka = _windows(a, m, dev)
    zb, okb = (za, oka) if b is None else _windows(b, m, dev)
    excl = m // 4 if b is None else 0
    if case["kind"] in ("selfjoin", "abjoin"):
        return _distance(_best(za, oka, zb, okb, excl), m).cpu().numpy(), None
    if case["kind"] == "abdevice":
        ra, rb = _best(za, oka, zb, okb, 0), _best(zb, okb, za, oka, 0)
        return (torch.where(ra < -1, torch.full_like(ra, -2.0), ra), None,
                torch.where(rb < -1, torch.full_like(rb, -2.0), rb), None)
    thr = case["threshold"]
    if case["kind"] == "sum":
        return torch.cat([torch.where(r > thr, r, torch.zeros_like(r)).sum(1)
                          for _, r in _corr_blocks(za, oka, zb, okb, excl)]).cpu().numpy()
    if case["kind"] == "knn":
        best = torch.cat([torch.topk(r, case["k"], dim=1).values
                          for _, r in _corr_blocks(za, oka, zb, okb, excl)])
        best = torch.where(best > thr, best, torch.full_like(best, -2.0))
        return best.reshape(-1).cpu().numpy(), None
    # matrix: the best cell above the diagonal's exclusion zone per grid entry
    # (rows: the smaller window index)
    side, ns = case["side"], za.shape[0]
    per = -(-ns // side)
    grid = torch.full((side, side), -2.0, dtype=torch.float64, device=dev)
    col = torch.arange(ns, device=dev)
    for i, r in _corr_blocks(za, oka, zb, okb, excl):
        rows = torch.arange(i, i + r.shape[0], device=dev)
        r.masked_fill_(col[None, :] < rows[:, None], -3.0)
        r = torch.nn.functional.pad(r, (0, per * side - ns), value=-3.0)
        cells = r.reshape(r.shape[0], side, per).max(2).values
        grid.scatter_reduce_(0, (rows // per)[:, None].expand(-1, side), cells, "amax")
    grid = torch.where(grid > thr, grid, torch.full_like(grid, -2.0))
    return _distance(grid, m).cpu().numpy()
