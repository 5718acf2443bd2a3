// join_fp64.cu -- the plain (all-FP64) form of the SCAMP join.
//
// Replaces the reference's do_tile (src/kernels.cu:22-167) and its tile
// scheduler (src/SCAMP.cpp:25-169, src/tile.cpp:546-707).  One persistent
// kernel walks a device-side work queue of units; a unit is a band of
// kFp64Band diagonals times two segments of seg_len rows (the segments run
// interleaved, which doubles the independent FP64 chains per thread).  Each
// segment starts from an FP64 direct-dot seed (the reference's QT seed,
// src/qt_helper.cpp:52-72), then every cell costs exactly four FP64-pipe
// instructions: two DFMA for the recurrence and two for r = cov*inv_c*inv_r.
// GB300 issues FP64 at 1/62 of its FP32 rate (measured), so everything else
// -- compares, index tracking, key packing -- runs on the integer pipe, which
// has ample spare issue slots.
//
// Profile updates follow the reference's semantics (strict '>' with NaN never
// winning, src/kernel_gpu_utils.h:138-179; SUM_THRESH adds r when r > thr,
// src/kernels_compute.h:88-113) but merge through order-preserving 64-bit
// keys: per-slab maxima are staged in shared memory and published with one
// global atomicMax per improved entry (the reference's packed-u64 CAS loop,
// src/kernel_gpu_utils.h:261-307, becomes a single atomic).
#include <cstdint>

#include "engine.cuh"

namespace scamp_gb300 {

namespace {

constexpr int kThreads = 128;
constexpr int kDiags = 4;             // diagonals per thread
constexpr int kBand = kThreads * kDiags;  // diagonals per unit
constexpr int kRows = 4;              // rows per step
constexpr int kSlab = 64;             // rows staged per slab
constexpr int kCols = kSlab + kBand;  // columns staged per slab

__device__ __forceinline__ double fmul_dfma(double a, double b) {
  // a*b issued as a DFMA with -0 addend (exact, keeps -0): on GB300 DFMA
  // retires faster than DMUL (measured).
  double r;
  asm("fma.rn.f64 %0, %1, %2, 0d8000000000000000;" : "=d"(r) : "d"(a), "d"(b));
  return r;
}

__device__ __forceinline__ uint64_t umax64(uint64_t a, uint64_t b) {
  return a > b ? a : b;
}

// Ordered integer image of a double; NaN maps below everything.
__device__ __forceinline__ int64_t ord_double(double x) {
  const int64_t b = __double_as_longlong(x);
  if ((b & 0x7FF0000000000000ll) == 0x7FF0000000000000ll) return INT64_MIN;
  return b ^ ((b >> 63) & 0x7FFFFFFFFFFFFFFFll);
}

// SUM_THRESH adds in fixed point: r as a signed integer in units of 2^-53
// (the last place of r in [1/2, 1); smaller ones rounded to it, not cut, which
// would take 2^-55 and more from every term), integer pipe only.  Integer sums are exact, so a slab's sum (at most 512 cells, |r| <= 1
// up to rounding: 2^62) carries less error than one added in FP64, and they
// leave the FP64 pipe the recurrence's four operations per cell: the two
// additions per cell and the row reductions' shuffles in FP64 had taken three
// quarters of the pipe (32768 samples, m = 128, r > 0.9: 14.1 -> 9.7 ms, and 4.8
// with the segments of fp64_rows(): 88% of the FP64 pipe).  A value beyond
// 1.5 (a recurrence that lost everything to a spike) counts as 1.5, so that
// no slab's sum can wrap around.
constexpr int kSumFrac = 53;
__device__ __forceinline__ long long fixed_r(double r) {
  const uint64_t bits = static_cast<uint64_t>(__double_as_longlong(r));
  const int e = static_cast<int>((bits >> 52) & 0x7FF);
  const uint64_t sig = (bits & 0x000FFFFFFFFFFFFFull) | (e ? (1ull << 52) : 0);
  const int s = 1075 - kSumFrac - e;  // |r| 2^53 = sig 2^-s
  constexpr uint64_t kMost = 3ull << (kSumFrac - 1);
  uint64_t mag = s >= 64 ? 0 : (s >= 0 ? (((sig << 1) >> s) + 1) >> 1 : (s == -1 ? sig << 1 : kMost));
  if (mag > kMost) mag = kMost;
  return (bits >> 63) ? -static_cast<long long>(mag) : static_cast<long long>(mag);
}
__device__ __forceinline__ double sum_of_fixed(unsigned long long v) {
  return static_cast<double>(static_cast<long long>(v)) * (1.0 / (1ull << kSumFrac));
}

struct SmemFp64 {
  double df_r[2][kSlab], dg_r[2][kSlab], iv_r[2][kSlab];
  double df_c[2][kCols], dg_c[2][kCols], iv_c[2][kCols];
  union {
    struct {
      unsigned long long col[2][kCols];
      unsigned long long row[2][kSlab];
    } key;
    struct {
      unsigned long long col[2][kCols];  // fixed point, two's complement
      unsigned long long row[2][kSlab];
    } sum;
  } prof;
  unsigned char dirty_col[2][kCols];
  unsigned char dirty_row[2][kSlab];
  long long unit;
};

// FP64 direct-dot seeds: the covariances of row window i with the column
// windows j .. j + kDiags - 1 (the reference's QT seed,
// src/qt_helper.cpp:52-72).  The row window is centred by its own mean, the
// column samples by the first window's, which the four windows share:
//   cov_k = sum x_t y_{t+k} - (mean_{j+k} - mean_j) sum x_t,
// 7 FP64 operations per sample for four windows against 9 with each window
// centred by itself.  The products then carry the means' difference, so each
// window is centred by itself where that exceeds 1/4 of a window's standard
// deviation in some lane of the warp (beside 1/4 it adds 3% to the rounding; a
// spike, or a gap on an offset, that leaves with the first window carries any
// amount), and where a window has no inverse norm to tell.  At 1/8 random
// walks cross it: 32768 samples, m = 128, 5.18 ms against 5.09, which it also
// takes without the test.  Windows at or past C.ns get 0.  Called by whole
// warps.
__device__ __forceinline__ void seed_fp64(const SeriesDev& R, const SeriesDev& C, int64_t i,
                                          int64_t j, int64_t m, double (&cov)[kDiags]) {
  const double mr = R.mean[i];
  double mc[kDiags];
  bool near = true;
#pragma unroll
  for (int k = 0; k < kDiags; ++k) {
    cov[k] = 0.0;
    mc[k] = j + k < C.ns ? C.mean[j + k] : 0.0;
    if (k > 0 && j + k < C.ns) {
      const double shift = (mc[k] - mc[0]) * C.inv[j + k];
      near = near && shift * shift * static_cast<double>(m) <= 1.0 / 16.0;
    }
  }
  near = __all_sync(0xffffffffu, near);
  if (j >= C.ns) return;
  const double* __restrict__ tr = R.T + i;
  const double* __restrict__ tc = C.T + j;
  const int64_t nc = C.n - j;  // column samples from j on
  const double shared = near ? mc[0] : 0.0;
  double xs = 0.0;
  double y[kDiags];
#pragma unroll
  for (int k = 0; k + 1 < kDiags; ++k) y[k] = k < nc ? tc[k] - shared : 0.0;
  if (near) {
#pragma unroll 4
    for (int64_t t = 0; t < m; ++t) {
      const double x = tr[t] - mr;
      y[kDiags - 1] = t + kDiags - 1 < nc ? tc[t + kDiags - 1] - shared : 0.0;
      xs += x;
#pragma unroll
      for (int k = 0; k < kDiags; ++k) cov[k] = fma(x, y[k], cov[k]);
#pragma unroll
      for (int k = 0; k + 1 < kDiags; ++k) y[k] = y[k + 1];
    }
#pragma unroll
    for (int k = 0; k < kDiags; ++k) cov[k] = fma(-(mc[k] - shared), xs, cov[k]);
  } else {
#pragma unroll 4
    for (int64_t t = 0; t < m; ++t) {
      const double x = tr[t] - mr;
      y[kDiags - 1] = t + kDiags - 1 < nc ? tc[t + kDiags - 1] : 0.0;
#pragma unroll
      for (int k = 0; k < kDiags; ++k) cov[k] = fma(x, y[k] - mc[k], cov[k]);
#pragma unroll
      for (int k = 0; k + 1 < kDiags; ++k) y[k] = y[k + 1];
    }
  }
#pragma unroll
  for (int k = 0; k < kDiags; ++k)
    if (j + k >= C.ns) cov[k] = 0.0;
}

}  // namespace

__global__ void __launch_bounds__(kThreads)
join_fp64_kernel(JoinParams P) {
  __shared__ SmemFp64 sm;
  const int t = threadIdx.x;
  const int lane = t & 31;
  const bool is_1nn = P.profile_type == 1;
  const double thr = P.threshold;
  const int64_t ord_thr = ord_double(thr);
  const int64_t K = P.seg_len;
  // The whole queue, or the units the exact form left: each in half bands
  // (its bands are twice as wide), and where they are too few for the
  // resident CTAs also in pieces of its rows (a CTA alone on an SM runs at a
  // quarter of the SM's FP64 rate: a handful of units of 1024 rows took 4.3
  // ms), each of at least 128 rows and m, which bounds the work of its seeds.
  const bool listed = P.fp64_list != nullptr;
  int64_t pieces = 1, piece_len = K, total_units = P.total_units;
  if (listed) {
    const int64_t left = static_cast<int64_t>(*P.fp64_count);
    const int64_t least = P.m > 128 ? P.m : 128;
    if (left > 0) pieces = gridDim.x / (2 * left);
    if (pieces > K / least) pieces = K / least;
    if (pieces < 1) pieces = 1;
    piece_len = ((K + pieces - 1) / pieces + kSlab - 1) / kSlab * kSlab;
    total_units = 2 * left * pieces;
  }

  for (;;) {
    if (t == 0) sm.unit = static_cast<long long>(atomicAdd(P.unit_counter, 1ull));
    __syncthreads();
    const int64_t u = sm.unit;
    __syncthreads();
    if (u >= total_units) break;

    int pi;
    int64_t band, ub;
    const int64_t half = u / pieces, row_off = (u - half * pieces) * piece_len;
    decode_unit(P, listed ? P.fp64_list[half >> 1] : u, &pi, &band, &ub);
    const Problem& pr = P.prob[pi];
    const int64_t D0 = pr.d_lo + band * P.band_width + (listed ? (half & 1) * kBand : 0);
    if (D0 >= pr.d_hi) continue;
    const int64_t rows_b = band_rows(pr.R.ns, pr.C.ns, D0);
    int64_t seg_row[2], seg_len[2];
    seg_row[0] = ub * 2 * K + row_off;
    seg_row[1] = seg_row[0] + K;
    const int64_t most = K - row_off < piece_len ? K - row_off : piece_len;
    for (int g = 0; g < 2; ++g) {
      int64_t l = rows_b - seg_row[g];
      seg_len[g] = l < 0 ? 0 : (l > most ? most : l);
    }
    const int64_t d_my = D0 + t * kDiags;

    // Seeds for this thread's diagonals.
    double cov[2][kDiags];
#pragma unroll
    for (int g = 0; g < 2; ++g) {
      if (seg_len[g] > 0) {
        seed_fp64(pr.R, pr.C, seg_row[g], seg_row[g] + d_my, P.m, cov[g]);
      } else {
#pragma unroll
        for (int k = 0; k < kDiags; ++k) cov[g][k] = 0.0;
      }
    }
    // Per-diagonal validity (diagonal range and the is_aligned exclusion).
    bool dvalid[kDiags];
    for (int k = 0; k < kDiags; ++k) {
      const int64_t d = d_my + k;
      dvalid[k] = d < pr.d_hi && !(d >= pr.x_lo && d < pr.x_hi);
    }

    const int64_t nslabs = (seg_len[0] + kSlab - 1) / kSlab;
    for (int64_t q = 0; q < nslabs; ++q) {
      // ---- stage rows, columns and profile entries of this slab ----
      for (int g = 0; g < 2; ++g) {
        const int64_t rbase = seg_row[g] + q * kSlab;
        const int64_t rend = seg_row[g] + seg_len[g];
        for (int x = t; x < kSlab; x += kThreads) {
          const int64_t i = rbase + x;
          const bool ok = i < rend;
          sm.df_r[g][x] = ok ? pr.R.df[i] : 0.0;
          sm.dg_r[g][x] = ok ? pr.R.dg[i] : 0.0;
          sm.iv_r[g][x] = ok ? pr.R.inv[i] : __longlong_as_double(0x7FF8000000000000ll);
          if (is_1nn) {
            sm.prof.key.row[g][x] = (ok && pr.key_row) ? pr.key_row[i] : 0ull;
          } else {
            sm.prof.sum.row[g][x] = 0ull;
          }
          sm.dirty_row[g][x] = 0;
        }
        const int64_t cbase = rbase + D0;
        for (int x = t; x < kCols; x += kThreads) {
          const int64_t j = cbase + x;
          const bool ok = j < pr.C.ns;
          sm.df_c[g][x] = ok ? pr.C.df[j] : 0.0;
          sm.dg_c[g][x] = ok ? pr.C.dg[j] : 0.0;
          sm.iv_c[g][x] = ok ? pr.C.inv[j] : __longlong_as_double(0x7FF8000000000000ll);
          if (is_1nn) {
            sm.prof.key.col[g][x] = (ok && pr.key_col) ? pr.key_col[j] : 0ull;
          } else {
            sm.prof.sum.col[g][x] = 0ull;
          }
          sm.dirty_col[g][x] = 0;
        }
      }
      __syncthreads();

      // ---- compute kSlab rows in steps of kRows ----
      for (int r0 = 0; r0 < kSlab; r0 += kRows) {
        const int cb = r0 + t * kDiags;  // first staged column of this step
        if (is_1nn) {
          uint64_t cbest[2][kDiags + kRows - 1];
          uint64_t rbest[2][kRows];
#pragma unroll
          for (int g = 0; g < 2; ++g) {
#pragma unroll
            for (int c = 0; c < kDiags + kRows - 1; ++c) cbest[g][c] = 0;
#pragma unroll
            for (int rr = 0; rr < kRows; ++rr) rbest[g][rr] = 0;
          }
#pragma unroll
          for (int g = 0; g < 2; ++g) {
            const int64_t row0 = seg_row[g] + q * kSlab + r0;
#pragma unroll
            for (int rr = 0; rr < kRows; ++rr) {
              const double dfr = sm.df_r[g][r0 + rr];
              const double dgr = sm.dg_r[g][r0 + rr];
              const double ivr = sm.iv_r[g][r0 + rr];
              const int64_t i = row0 + rr;
#pragma unroll
              for (int k = 0; k < kDiags; ++k) {
                const int c = cb + rr + k;
                const double r = fmul_dfma(fmul_dfma(cov[g][k], sm.iv_c[g][c]), ivr);
                uint64_t qv = q_from_double_bits(__double_as_longlong(r), P.kl.frac_bits);
                if (!dvalid[k]) qv = 0;
                const int64_t j = i + d_my + k;
                rbest[g][rr] = umax64(rbest[g][rr], make_key(qv, j, P.kl));
                cbest[g][rr + k] = umax64(cbest[g][rr + k], make_key(qv, i, P.kl));
                cov[g][k] = fma(sm.df_c[g][c], dgr, cov[g][k]);
                cov[g][k] = fma(dfr, sm.dg_c[g][c], cov[g][k]);
              }
            }
          }
          // publish column maxima to shared memory
          if (pr.key_col) {
#pragma unroll
            for (int g = 0; g < 2; ++g) {
#pragma unroll
              for (int c = 0; c < kDiags + kRows - 1; ++c) {
                const uint64_t v = cbest[g][c];
                unsigned long long* slot = &sm.prof.key.col[g][cb + c];
                if (v > *slot) {
                  if (atomicMax(slot, static_cast<unsigned long long>(v)) < v)
                    sm.dirty_col[g][cb + c] = 1;
                }
              }
            }
          }
          // row maxima: warp reduction, then one shared atomic per warp
          if (pr.key_row) {
#pragma unroll
            for (int g = 0; g < 2; ++g) {
#pragma unroll
              for (int rr = 0; rr < kRows; ++rr) {
                uint64_t v = rbest[g][rr];
#pragma unroll
                for (int o = 16; o > 0; o >>= 1)
                  v = umax64(v, __shfl_xor_sync(0xffffffffu, v, o));
                if (lane == 0) {
                  unsigned long long* slot = &sm.prof.key.row[g][r0 + rr];
                  if (v > *slot) {
                    if (atomicMax(slot, static_cast<unsigned long long>(v)) < v)
                      sm.dirty_row[g][r0 + rr] = 1;
                  }
                }
              }
            }
          }
        } else {
          // SUM_THRESH: sum r over cells with r > threshold.
          unsigned long long csum[2][kDiags + kRows - 1];
          unsigned long long rsum[2][kRows];
#pragma unroll
          for (int g = 0; g < 2; ++g) {
#pragma unroll
            for (int c = 0; c < kDiags + kRows - 1; ++c) csum[g][c] = 0;
#pragma unroll
            for (int rr = 0; rr < kRows; ++rr) rsum[g][rr] = 0;
          }
#pragma unroll
          for (int g = 0; g < 2; ++g) {
#pragma unroll
            for (int rr = 0; rr < kRows; ++rr) {
              const double dfr = sm.df_r[g][r0 + rr];
              const double dgr = sm.dg_r[g][r0 + rr];
              const double ivr = sm.iv_r[g][r0 + rr];
#pragma unroll
              for (int k = 0; k < kDiags; ++k) {
                const int c = cb + rr + k;
                const double r = fmul_dfma(fmul_dfma(cov[g][k], sm.iv_c[g][c]), ivr);
                const bool take = dvalid[k] && ord_double(r) > ord_thr;
                const unsigned long long v =
                    take ? static_cast<unsigned long long>(fixed_r(r)) : 0ull;
                rsum[g][rr] += v;
                csum[g][rr + k] += v;
                cov[g][k] = fma(sm.df_c[g][c], dgr, cov[g][k]);
                cov[g][k] = fma(dfr, sm.dg_c[g][c], cov[g][k]);
              }
            }
          }
          if (pr.sum_col) {
#pragma unroll
            for (int g = 0; g < 2; ++g)
#pragma unroll
              for (int c = 0; c < kDiags + kRows - 1; ++c)
                if (csum[g][c] != 0) atomicAdd(&sm.prof.sum.col[g][cb + c], csum[g][c]);
          }
          if (pr.sum_row) {
#pragma unroll
            for (int g = 0; g < 2; ++g)
#pragma unroll
              for (int rr = 0; rr < kRows; ++rr) {
                unsigned long long v = rsum[g][rr];
#pragma unroll
                for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
                if (lane == 0 && v != 0) atomicAdd(&sm.prof.sum.row[g][r0 + rr], v);
              }
          }
        }
      }
      __syncthreads();

      // ---- publish the slab's improved entries to the global profile ----
      for (int g = 0; g < 2; ++g) {
        const int64_t rbase = seg_row[g] + q * kSlab;
        const int64_t rend = seg_row[g] + seg_len[g];
        const int64_t cbase = rbase + D0;
        if (is_1nn) {
          if (pr.key_col)
            for (int x = t; x < kCols; x += kThreads)
              if (sm.dirty_col[g][x] && cbase + x < pr.C.ns)
                atomicMax(reinterpret_cast<unsigned long long*>(&pr.key_col[cbase + x]),
                          sm.prof.key.col[g][x]);
          if (pr.key_row)
            for (int x = t; x < kSlab; x += kThreads)
              if (sm.dirty_row[g][x] && rbase + x < rend)
                atomicMax(reinterpret_cast<unsigned long long*>(&pr.key_row[rbase + x]),
                          sm.prof.key.row[g][x]);
        } else {
          if (pr.sum_col)
            for (int x = t; x < kCols; x += kThreads) {
              const double v = sum_of_fixed(sm.prof.sum.col[g][x]);
              if (v != 0.0 && cbase + x < pr.C.ns) atomicAdd(&pr.sum_col[cbase + x], v);
            }
          if (pr.sum_row)
            for (int x = t; x < kSlab; x += kThreads) {
              const double v = sum_of_fixed(sm.prof.sum.row[g][x]);
              if (v != 0.0 && rbase + x < rend) atomicAdd(&pr.sum_row[rbase + x], v);
            }
        }
      }
      __syncthreads();
    }
  }
}

int fp64_band_width() { return kBand; }
int fp64_slab_rows() { return kSlab; }
int fp64_threads() { return kThreads; }

}  // namespace scamp_gb300
