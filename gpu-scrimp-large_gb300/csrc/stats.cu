// stats.cu -- window statistics on device, in compensated FP64.
//
// Replaces the reference's host-side, sequential precompute
// (src/cpu_stats.cpp:11-160, called from src/SCAMP.cpp:195-206) with one
// kernel.  Each warp owns kStatsChunk consecutive windows: it sums its first
// window directly, then the others from it (the reference's rolling,
// TwoSum-compensated update, as scans over the warp's lanes), so the rounding
// error restarts every kStatsChunk windows instead of growing over the whole
// series.  ULTRA precision sums every window directly (the reference's
// brute-force O(nm) option, src/cpu_stats.cpp:31-41, 85-97).
//
// Semantics kept exactly:
//  - non-finite samples become 0 and poison every window holding them
//    (src/cpu_stats.cpp:11-29);
//  - invnorm = 1/sqrt(ssd), NaN when the window held a non-finite sample or
//    ssd <= 1e-13 (src/cpu_stats.cpp:140-152);
//  - df[i] = (T[i+m]-T[i])/2, dg[i] = (T[i+m]-mu[i+1]) + (T[i]-mu[i]), and
//    df = dg = 0 at the last window (src/cpu_stats.cpp:154-157).
#include <cmath>

#include "engine.cuh"

namespace scamp_gb300 {

namespace {

constexpr double kFlatnessEpsilon = 1e-13;  // src/cpu_stats.cpp:4

__device__ __forceinline__ double clean(double x) {
  return isfinite(x) ? x : 0.0;
}

// TwoSum accumulate (Knuth): s + c += x.
__device__ __forceinline__ void acc2(double& s, double& c, double x) {
  const double t = s + x;
  const double z = t - s;
  c += (s - (t - z)) + (x - z);
  s = t;
}

}  // namespace

// Sum of two compensated sums: (s, c) += (s2, c2).
__device__ __forceinline__ void add2(double& s, double& c, double s2, double c2) {
  acc2(s, c, s2);
  c += c2;
}

// One window's outputs from its mean (mu + mu_lo), the next window's mean
// and its sum of squared deviations.
struct StatsOut {
  double *mean, *inv, *df, *dg;
  float *mu_rel, *inv32, *df32, *dg32;
  float vmax, imax;  // the lane's largest |value| and inverse norm
};
__device__ __forceinline__ void write_window(StatsOut& o, int64_t w, double x_out, double x_in,
                                             bool has_next, double mu, double mu_lo, double mu_next,
                                             double mu_next_lo, double ssd, bool nan_window,
                                             double block_off) {
  const double iv = (nan_window || !(ssd > kFlatnessEpsilon)) ? nan("") : 1.0 / sqrt(ssd);
  double f = 0, g = 0;
  if (has_next) {
    f = (x_in - x_out) / 2.0;
    g = ((x_in - mu_next) - mu_next_lo) + ((x_out - mu) - mu_lo);
  }
  const float mr = static_cast<float>((mu - block_off) + mu_lo);
  const float iv32 = static_cast<float>(iv), f32 = static_cast<float>(f), g32 = static_cast<float>(g);
  o.mean[w] = mu;
  o.mu_rel[w] = mr;
  o.inv[w] = iv;
  o.df[w] = f;
  o.dg[w] = g;
  o.inv32[w] = iv32;
  o.df32[w] = f32;
  o.dg32[w] = g32;
  o.vmax = fmaxf(fmaxf(o.vmax, fabsf(mr)), fmaxf(fabsf(f32), fabsf(g32)));
  o.imax = fmaxf(o.imax, iv32);  // NaN (no match possible) does not count
}

// Statistics of windows [chunk * kStatsChunk, (chunk + 1) * kStatsChunk) of
// one series, by one warp (every lane calls it; `lane` its lane).
//
// The lanes share the direct sums of the chunk's first window (each sums
// every 32nd sample, compensated; the partial sums meet in a shuffle tree).
// Window w's sum is the first window's plus the differences x[v + m] - x[v],
// v < w, and its sum of squares the first window's plus the reference's
// recurrence terms (src/cpu_stats.cpp:114-117): both are compensated scans
// over the lanes, 32 windows at a time.  Per window that leaves one
// divide and one square root per lane and no chain from window to window.
// Bound by the FP64 pipe: 2 m x 8 additions per 64 windows plus about 100
// per window.  One thread per 64-window chunk, which this replaces, was bound by
// its own chain of FP64 latencies at every size: 276 / 348 / 1158 us at 1000
// (m = 50) / 131072 (m = 100) / 40009 samples (m = 1024).
__device__ __forceinline__ void stats_body(int64_t chunk, int lane, const double* __restrict__ T_raw,
                                           int64_t n, int64_t m, int ultra, int bshift,
                                           double* __restrict__ T_clean, float* __restrict__ T32,
                                           float* __restrict__ bhi, float* __restrict__ blo,
                                           StatsOut& o) {
  constexpr unsigned kAll = 0xffffffffu;
  const int64_t ns = n - m + 1;
  const int64_t w0 = chunk * kStatsChunk;
  if (w0 >= ns) return;
  const int64_t w1 = (w0 + kStatsChunk < ns) ? w0 + kStatsChunk : ns;

  // Cleaned samples owned by this chunk (the last chunk also owns the tail).
  // Block offsets are the blocks' first (cleaned) samples.
  auto block_off = [&](int64_t b) { return clean(T_raw[b << bshift]); };
  {
    const int64_t s_end = (w1 == ns) ? n : w1;
    for (int64_t t = w0 + lane; t < s_end; t += 32) {
      const double c = clean(T_raw[t]);
      T_clean[t] = c;
      const int64_t b = t >> bshift;
      const double off = block_off(b);
      const float rel = static_cast<float>(c - off);
      T32[t] = rel;
      o.vmax = fmaxf(o.vmax, fabsf(rel));
      if ((b << bshift) == t) {
        const float hi = static_cast<float>(off);
        bhi[b] = hi;
        blo[b] = static_cast<float>(off - static_cast<double>(hi));
      }
    }
  }

  // The mean is carried as mu + mu_lo: the low part restores the digits the
  // division drops, which matters for series with a large offset relative
  // to their variation (dg subtracts the mean from the raw samples).
  const double md = static_cast<double>(m);
  auto mean_of = [&](double ps, double pc, double& mu, double& mu_lo) {
    mu = (ps + pc) / md;
    mu_lo = (fma(-mu, md, ps) + pc) / md;
  };

  if (ultra) {
    // every window summed directly, in order, by its own lane
    for (int64_t w = w0 + lane; w < w1; w += 32) {
      double ps = 0, pc = 0;
      bool bad = false;
      for (int64_t t = 0; t < m; ++t) {
        const double x = T_raw[w + t];
        bad = bad || !isfinite(x);
        acc2(ps, pc, clean(x));
      }
      double mu, mu_lo, mu_next = 0, mu_next_lo = 0;
      mean_of(ps, pc, mu, mu_lo);
      double ss = 0, sc = 0;
      for (int64_t t = 0; t < m; ++t) {
        const double v = clean(T_raw[w + t]) - mu;
        acc2(ss, sc, v * v);
      }
      const bool has_next = w + 1 < ns;
      if (has_next) {
        double s2 = 0, c2 = 0;
        for (int64_t t = 0; t < m; ++t) acc2(s2, c2, clean(T_raw[w + 1 + t]));
        mean_of(s2, c2, mu_next, mu_next_lo);
      }
      write_window(o, w, clean(T_raw[w]), has_next ? clean(T_raw[w + m]) : 0.0, has_next, mu, mu_lo,
                   mu_next, mu_next_lo, ss + sc, bad, block_off(w >> bshift));
    }
    return;
  }

  // Window w0: sum, mean, sum of squared deviations, last non-finite sample.
  double ps = 0, pc = 0;
  int64_t last_bad = -1;
  for (int64_t t = lane; t < m; t += 32) {
    const double x = T_raw[w0 + t];
    if (!isfinite(x)) last_bad = w0 + t;
    acc2(ps, pc, clean(x));
  }
#pragma unroll
  for (int s = 16; s > 0; s >>= 1) {
    add2(ps, pc, __shfl_xor_sync(kAll, ps, s), __shfl_xor_sync(kAll, pc, s));
    const int64_t ob = __shfl_xor_sync(kAll, last_bad, s);
    last_bad = ob > last_bad ? ob : last_bad;
  }
  // (the tree adds in an order that depends on the lane: one lane's result)
  ps = __shfl_sync(kAll, ps, 0);
  pc = __shfl_sync(kAll, pc, 0);
  double mu0, mu0_lo;
  mean_of(ps, pc, mu0, mu0_lo);
  double ss = 0, sc = 0;
  for (int64_t t = lane; t < m; t += 32) {
    // (x - mu)^2 as a compensated product too: what a spike in window w0
    // rounds stays in the sums after it has left.  (With vl^2: it is m times
    // the square of the mean's rounding, 6e-11 of the sum for noise of 0.01 on
    // an offset of 1e9.)
    double vh = clean(T_raw[w0 + t]), vl = 0;
    acc2(vh, vl, -mu0);
    vl -= mu0_lo;
    const double p = vh * vh;
    sc += fma(vl, fma(2.0, vh, vl), fma(vh, vh, -p));
    acc2(ss, sc, p);
  }
#pragma unroll
  for (int s = 16; s > 0; s >>= 1)
    add2(ss, sc, __shfl_xor_sync(kAll, ss, s), __shfl_xor_sync(kAll, sc, s));
  ss = __shfl_sync(kAll, ss, 0);
  sc = __shfl_sync(kAll, sc, 0);

  // 32 windows at a time; (ps, pc) and (ss, sc) are those of window wb.
  int top = 0;  // high word of the chunk's largest sum of squares so far
  for (int64_t wb = w0; wb < w1; wb += 32) {
    const int64_t w = wb + lane;
    const bool active = w < w1;
    const bool has_next = w + 1 < ns;
    const double x_out = active ? clean(T_raw[w]) : 0.0;
    const double x_raw = (active && has_next) ? T_raw[w + m] : 0.0;
    const double x_in = clean(x_raw);
    // sums of windows wb + 1 .. wb + 32: inclusive scan of the differences
    double ds = 0, dc = 0;
    acc2(ds, dc, x_in);
    acc2(ds, dc, -x_out);
#pragma unroll
    for (int s = 1; s < 32; s <<= 1) {
      const double us = __shfl_up_sync(kAll, ds, s), uc = __shfl_up_sync(kAll, dc, s);
      if (lane >= s) add2(ds, dc, us, uc);
    }
    double ns_s = ps, ns_c = pc;  // the sum of window w + 1
    add2(ns_s, ns_c, ds, dc);
    double mu_next, mu_next_lo;
    mean_of(ns_s, ns_c, mu_next, mu_next_lo);
    double mu = __shfl_up_sync(kAll, mu_next, 1), mu_lo = __shfl_up_sync(kAll, mu_next_lo, 1);
    if (lane == 0) {
      mu = mu0;
      mu_lo = mu0_lo;
    }
    // Sums of squares: the recurrence's terms with the means' low parts, so
    // that a large offset's rounded mean does not leave a per-step residue
    // (b - a)(delta_w + delta_w+1).  Each term is a compensated product: one
    // rounding of a spike's term would stay in every later sum of the chunk
    // (2^-53 of the spike's square, 1e-6 of the norm behind a spike of 10^6
    // standard deviations).
    double es = 0, ec = 0;
    if (active && has_next) {
      double ph = 0, pl = 0, qh = 0, ql = 0;
      acc2(ph, pl, x_out);
      acc2(ph, pl, -mu);
      acc2(ph, pl, x_in);
      acc2(ph, pl, -mu_next);
      pl -= mu_lo + mu_next_lo;
      acc2(qh, ql, x_in);
      acc2(qh, ql, -x_out);
      es = ph * qh;
      ec = fma(ph, qh, -es) + fma(ph, ql, pl * qh);
    }
#pragma unroll
    for (int s = 1; s < 32; s <<= 1) {
      const double us = __shfl_up_sync(kAll, es, s), uc = __shfl_up_sync(kAll, ec, s);
      if (lane >= s) add2(es, ec, us, uc);
    }
    double nss = ss, nsc = sc;  // of window w + 1
    add2(nss, nsc, es, ec);
    double ssd_s = __shfl_up_sync(kAll, nss, 1), ssd_c = __shfl_up_sync(kAll, nsc, 1);
    if (lane == 0) {
      ssd_s = ss;
      ssd_c = sc;
    }
    // the last non-finite sample of window w: one in front of sample w + m,
    // or the chunk's running one
    const unsigned bad = __ballot_sync(kAll, active && has_next && !isfinite(x_raw));
    const unsigned before = bad & ((1u << lane) - 1u);
    int64_t lb = last_bad;
    if (before) lb = wb + m + (31 - __clz(before));
    double ssd = ssd_s + ssd_c;
    top = max(top, static_cast<int>(__reduce_max_sync(
                       kAll, active ? static_cast<unsigned>(max(__double2hiint(ssd), 0)) : 0u)));
    if (active) {
      // Summed again directly, so that no accumulated residue shows: a
      // near-flat ssd (for the flatness rule), and one 2^40 below the largest
      // of its chunk, of which the recurrence keeps 2^-104 (unit noise, m =
      // 100, behind a spike of 1e10 349 u of the ssd, of 1e14 2.5e-6; now 2^-64
      // of it at most).
      if (ssd <= 1e3 * kFlatnessEpsilon || (top >> 20) - (__double2hiint(ssd) >> 20) > 40) {
        double s2 = 0, c2 = 0;
        for (int64_t t = 0; t < m; ++t) {
          const double v = (clean(T_raw[w + t]) - mu) - mu_lo;
          acc2(s2, c2, v * v);
        }
        ssd = s2 + c2;
      }
      write_window(o, w, x_out, x_in, has_next, mu, mu_lo, mu_next, mu_next_lo, ssd, lb >= w,
                   block_off(w >> bshift));
    }
    // window wb + 32
    ps = __shfl_sync(kAll, ns_s, 31);
    pc = __shfl_sync(kAll, ns_c, 31);
    ss = __shfl_sync(kAll, nss, 31);
    sc = __shfl_sync(kAll, nsc, 31);
    mu0 = __shfl_sync(kAll, mu_next, 31);
    mu0_lo = __shfl_sync(kAll, mu_next_lo, 31);
    if (bad) last_bad = wb + m + (31 - __clz(bad));
  }
}

__global__ void __launch_bounds__(kStatsThreads) stats_kernel(StatsJob j, int ultra) {
  const int64_t warp = (static_cast<int64_t>(blockIdx.x) * kStatsThreads + threadIdx.x) >> 5;
  StatsOut o{j.mean, j.inv, j.df, j.dg, j.mu_rel, j.inv32, j.df32, j.dg32, 0.f, 0.f};
  stats_body(warp, threadIdx.x & 31, j.T_raw, j.n, j.m, ultra, j.bshift, j.T_clean, j.T32, j.bhi,
             j.blo, o);
  if (j.range) {
    // non-negative floats order as their bits (an infinity counts as such)
    const unsigned v = __reduce_max_sync(0xffffffffu, __float_as_uint(o.vmax));
    const unsigned i = __reduce_max_sync(0xffffffffu, __float_as_uint(o.imax));
    if ((threadIdx.x & 31) == 0) {
      atomicMax(j.range, v);
      atomicMax(j.range + 1, i);
    }
  }
}

__global__ void __launch_bounds__(kStatsThreads)
stats_batch_kernel(const StatsJob* __restrict__ jobs, const int64_t* __restrict__ block_prefix,
                   int njobs) {
  const int64_t b = blockIdx.x;
  int lo = 0, hi = njobs;
  while (hi - lo > 1) {
    const int mid = (lo + hi) >> 1;
    if (block_prefix[mid] <= b) lo = mid; else hi = mid;
  }
  const StatsJob& j = jobs[lo];
  const int64_t warp = ((b - block_prefix[lo]) * kStatsThreads + threadIdx.x) >> 5;
  StatsOut o{j.mean, j.inv, j.df, j.dg, j.mu_rel, j.inv32, j.df32, j.dg32, 0.f, 0.f};
  stats_body(warp, threadIdx.x & 31, j.T_raw, j.n, j.m, 0, j.bshift, j.T_clean, j.T32, j.bhi, j.blo,
             o);
}

// ULTRA's update terms (the reference's compute_combined_stats_cpu,
// src/cpu_stats.cpp:162-196, used by src/tile.cpp:404-409).  With the
// covariance written against a constant c for one window,
//   cov(i+1, j+1) = cov(i, j) + (x[i+m] - mu[i+1]) (y[j+m] - c)
//                             - (x[i] - mu[i]) (y[j] - c),
// exact for c = mean(y[j+1 .. j+m-1]), the (m-1)-sample mean.  One side of a
// band takes the "A" terms of its series,
//   df = -(x[i] - mu[i]),  dg = x[i+m] - mu[i+1],
// the other the "B" terms,
//   df = y[j+m] - mu'[j+1],  dg = y[j] - mu'[j+1],
// so that df_c dg_r + df_r dg_c is the update above.  mu' is summed directly
// per window (TwoSum-compensated).  The last window's terms are 0 (the
// recurrence never leaves it).
__global__ void combined_stats_kernel(const double* __restrict__ T, int64_t n, int64_t m,
                                      const double* __restrict__ mean, int role_b,
                                      double* __restrict__ df, double* __restrict__ dg) {
  const int64_t ns = n - m + 1;
  const int64_t i = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
  if (i >= ns) return;
  if (i == ns - 1) {
    df[i] = 0.0;
    dg[i] = 0.0;
    return;
  }
  if (!role_b) {
    df[i] = -(T[i] - mean[i]);
    dg[i] = T[i + m] - mean[i + 1];
    return;
  }
  double s = 0.0, c = 0.0;
  for (int64_t t = i + 1; t < i + m; ++t) acc2(s, c, T[t]);
  const double mu1 = (s + c) / static_cast<double>(m - 1);
  df[i] = T[i + m] - mu1;
  dg[i] = T[i] - mu1;
}

}  // namespace scamp_gb300
