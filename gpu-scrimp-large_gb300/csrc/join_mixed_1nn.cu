// join_mixed_1nn.cu -- the mixed-precision band kernel: FP32 filter over an
// FP32 recurrence, exact path for the blocks it flags.  One body:
// 1NN_INDEX and SUM_THRESH in the mixed form (each with a per-cell and a
// per-step-bound filter), APPROX_ALL_NEIGHBORS (k-best lists) and MATRIX_SUMMARY,
// and the exact form of all but sums for DOUBLE joins (per-cell filter).
//
// Work decomposition as in join_fp64.cu (persistent kernel over a device
// queue of units = band of kBand diagonals x two row segments of seg_len
// rows; every thread advances kDiags diagonals in both segments as packed
// f32x2 pairs, .x = first segment, .y = second).
//
// Per cell the hot loop issues exactly the reference's arithmetic
// (src/kernels_compute.h:425-435): two FMAs advance the covariance and two
// multiplies form r = cov * invnorm_col * invnorm_row -- as f32x2 pair
// instructions, so the FP32 pipe, not the issue slot, bounds the loop.  What
// the reference does per cell on top of that -- compare, select, index
// bookkeeping (src/kernels_compute.h:25-113) -- is reduced to one running
// maximum of the whole 8x8x2 block per thread (3-input max.f32, two cells per
// instruction).
//
// 1NN_INDEX: a block whose maximum could beat the smallest best-so-far among
// its rows and columns, less an error margin, is queued for the exact path.
// The margin bounds the FP32 drift since the diagonal's anchor: per diagonal
// the kernel accumulates cov^2 and per thread the squared bound of the
// increments |df_c dg_r| + |df_r dg_c|, and uses
//   margin = C * 2^-24 * sqrt(rows * (sum cov^2 + sum inc^2)) * inv_c * inv_r.
// Each warp drains its queue cooperatively (8 lanes per queued block, both
// segments of a diagonal per lane as an f32x2 pair): cells that may improve
// their row or column are published with their FP32 value when the margin is
// below kTrust; otherwise the lower bound r - margin is published and the
// cell goes to a request buffer that verify_requests_kernel settles after the
// join with a direct dot product of the two centred windows.  The k-best
// form filters at each window's k-th best and inserts into its lists instead.
//
// 1NN in double precision (join_exact_1nn_kernel): the same walk, but the
// FP32 value only rules cells out.  In place of the margin every thread keeps
// a deterministic bound E on its covariances' error (kStepCov below); a cell
// whose r + E inv_c inv_r reaches its row's or column's best becomes a
// request, its lower bound raises the bests, and verify_exact_kernel computes
// every request that the final bests leave open in FP64.  Nothing FP32 is
// reported.  The profile is the FP64 kernel's at the FP32 kernel's rate:
// GB300 issues FP64 at 1/62 of FP32 and both forms cost 4 operations per
// cell (self-join of 131072 samples, m = 100: 67.5 -> 2.6 ms in the join
// kernels; 40009 samples with gaps, m = 1024: 39.0 -> 3.4 ms).
//
// Bounds pass (bound_exact_1nn_kernel), before double 1NN joins: from
// nothing, a window's best rises about ln(cells) times and every rise flags
// its whole 8 x 8 x 2 block, so after k cells per window about 640 / k of the
// steps are flagged, and a flagged step costs 30 plain ones: below some 10^5
// samples the exact path was most of the join (76-98% of the steps of
// 8000-20000 samples).  The pass walks every 2^14 / ns-th band first, each
// cell a multiply and a maximum more than the plain filter, and leaves every
// window a lower bound of its best over 2^14 cells; the join then flags 0.4 -
// 5% of its steps.  Device time: 10007 samples m = 100 0.79 -> 0.29 ms, 20000
// samples 0.76 -> 0.45 ms.  Mixed joins go without it: of two cells with equal
// FP32 values the first one published is the partner, and filters that start
// high let another one be first (81 of 8937 windows of a noisy sine, m = 64).
//
// SUM_THRESH (the reference's sum of every r above the threshold,
// src/kernels_compute.h:87-113 and 380-392), join_mixed_sum_kernel: every
// cell is decided in the main loop.  A cell above the threshold by more than
// the step's margin adds its FP32 r to its row's and its column's slab sums
// in shared memory (flushed to the FP64 profile by atomicAdd when the row's
// slab ends or the column leaves the column ring); the rare cells within the
// margin are settled by their own margin (sum_near): by the FP32 r within
// kTrust, else by a verification request that verify_requests_kernel adds if
// its directly computed r is above the threshold.
//
// MATRIX_SUMMARY: each thread keeps the running maximum of the grid entry its
// blocks fall in and publishes it when they move on (mat_cells_block routes
// the cells of a block that crosses a grid boundary).
//
// Anchors and verifications read an FP32 copy of each series stored relative
// to local block offsets (stats.cu), with every factor centred by its
// window's mean, so FP32 keeps its precision wherever the series wanders.
#include <cstdint>

#include "engine.cuh"

namespace scamp_gb300 {

namespace {

constexpr int kThreads = 128;
constexpr int kWarps = kThreads / 32;
constexpr int kDiags = 8;
constexpr int kBand = kThreads * kDiags;  // 1024 diagonals per unit
constexpr int kRows = 8;                  // rows per step
constexpr int kSlab = 128;                // rows staged per slab
constexpr int kSteps = kSlab / kRows;
constexpr int kCols = kSlab + kBand;      // staged columns per slab
constexpr int kBlocks = kCols / 8;        // 8-column blocks
// The staged columns form a ring over the unit's rows: slab q holds unit
// columns 128 q .. 128 q + kCols - 1 at ring columns (128 q + c) mod kCols, so
// a slab stages only the kSlab columns entering it.  Ring columns
// 0 .. kGhost - 1 are repeated after the end, so that a step's 15-column
// window never wraps.
constexpr int kGhost = 16;
constexpr int kPadG = kCols + kGhost + (kCols + kGhost) / 8;
constexpr int kAnchorChunk = 512;         // row-window samples per anchor pass
constexpr int kYSpan = kBand + kAnchorChunk + 16;     // staged column samples
constexpr int kYPad = (kYSpan / 8) * 10;              // padded: 10 pairs per 8
// blocks hold >= 32 samples: the span plus the block after its end
constexpr int kSpanBlk = kYSpan / 32 + 3;
constexpr int kQueue = 16;                // queued blocks per warp
constexpr int kReqChunk = 64;             // request slots a warp takes at a time (exact form)
constexpr float kEps = 5.9604645e-8f;     // 2^-24
constexpr float kBoundC = 4.0f;
// kBoundC * kEps * sqrt(kRows), widened by 2^-16 (see the step's threshold)
static_assert(kRows == 8, "kStepMarginC holds sqrt(8)");
constexpr float kStepMarginC = kBoundC * kEps * 2.8284271f * 1.0000153f;
// A candidate whose drift margin exceeds kTrust is verified by a direct dot
// product.  The margin is a statistical bound; 5e-6 leaves room for it to be
// exceeded (measured: max |r| error 6.6e-6 at 2048 rows per anchor, where
// kTrust = 8e-6 let one cell reach 1.07e-5).
constexpr float kTrust = 5e-6f;
constexpr float kNoTarget = 3.0e38f;      // best of a side that is not computed

// The exact form's error bounds (a deterministic bound E on |FP32 covariance
// - exact covariance| per thread and segment, first order in u = kEps with
// the factors below covering the higher orders and the bound's own FP32
// rounding):
//  - a step of 8 rows: each row rounds twice at no more than the largest
//    |cov| of the step's start plus the increments so far (16 u max|cov| +
//    72 u inc), and df, dg are rounded to FP32 (2 u per product, 16 u inc),
//    inc bounding |df_c dg_r| + |df_r dg_c| over the step's cells;
//  - an anchor: see anchor_bound().
// kBoundSlack widens E where it is used (its own sum of up to 2^17 terms
// rounds by less than 1%); kAbsSlack covers the roundings of r itself and of
// the comparisons (about 6 u of values within [-3, 1]).
constexpr float kStepCov = 16.0f * kEps;
constexpr float kStepInc = 88.0f * kEps;
constexpr float kBoundSlack = 1.01f;
constexpr float kAbsSlack = 1.0e-6f;
// A request whose bound is wider says that FP32 carries nothing there (a
// large step has passed through the windows); JoinParams::wide_budget.
constexpr float kWideBound = 1.0f / 8.0f;

typedef unsigned long long u64;

__device__ __forceinline__ u64 f2u(float2 v) {
  return (static_cast<u64>(__float_as_uint(v.y)) << 32) | __float_as_uint(v.x);
}
__device__ __forceinline__ float2 u2f(u64 v) {
  return make_float2(__uint_as_float(static_cast<uint32_t>(v)),
                     __uint_as_float(static_cast<uint32_t>(v >> 32)));
}
__device__ __forceinline__ float2 fma2(float2 a, float2 b, float2 c) {
  u64 d;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(f2u(a)), "l"(f2u(b)), "l"(f2u(c)));
  return u2f(d);
}
__device__ __forceinline__ float2 mul2(float2 a, float2 b) {
  u64 d;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(f2u(a)), "l"(f2u(b)));
  return u2f(d);
}
__device__ __forceinline__ float max3(float a, float b, float c) {
  float d;
  asm("max.f32 %0, %1, %2, %3;" : "=f"(d) : "f"(a), "f"(b), "f"(c));
  return d;
}
__device__ __forceinline__ float min3(float a, float b, float c) {
  float d;
  asm("min.f32 %0, %1, %2, %3;" : "=f"(d) : "f"(a), "f"(b), "f"(c));
  return d;
}
// PTX sqrt.approx.f32: an approximate square root (a few ulp); sqrt(0) = 0.
__device__ __forceinline__ float sqrt_approx(float x) {
  float r;
  asm("sqrt.approx.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
}
__device__ __forceinline__ float qnan() { return __int_as_float(0x7FC00000); }

// Largest |cov| over the 8 diagonals, per segment (NaN entries ignored).
__device__ __forceinline__ float2 absmax8(const float2 (&c)[8]) {
  float x = max3(fabsf(c[0].x), fabsf(c[1].x), fabsf(c[2].x));
  float y = max3(fabsf(c[0].y), fabsf(c[1].y), fabsf(c[2].y));
  x = max3(x, fabsf(c[3].x), fabsf(c[4].x));
  y = max3(y, fabsf(c[3].y), fabsf(c[4].y));
  x = max3(x, fabsf(c[5].x), fabsf(c[6].x));
  y = max3(y, fabsf(c[5].y), fabsf(c[6].y));
  return make_float2(fmaxf(x, fabsf(c[7].x)), fmaxf(y, fabsf(c[7].y)));
}

// A block queued for the exact path: the owner's covariances at the END of
// the step (the drain rewinds them), the step's drift estimate (largest
// sum cov^2 over the owner's diagonals plus the increment bound) and the
// block's position.
struct SlowItem {
  float2 cov[kDiags];  // covariances after the item's last step
  float2 vw;
  int s;      // first step within the slab | number of steps (1 or 2) << 8 |
              // segments to walk << 16 (bits 0-1 first step, 2-3 second)
  int owner;  // thread index of the owner
};

// CTA-uniform context of the exact path, kept in shared memory.
struct SlowCtx {
  const Problem* pr;
  uint64_t *key_row, *key_col;  // the problem's
  int64_t rbase[2];
  int64_t D0;  // first diagonal of the unit; thread t owns D0 + t*kDiags ..
  int ring0;   // ring column of the slab's first staged column
  // SUM_THRESH: cells with r > thr add r to their row's and column's sums
  // (r_best / c_best hold the slab's float sums instead of bests)
  bool sum_mode;
  float thr;
  int64_t m;
  KeyLayout kl;
  int prob;                        // index of the problem in JoinParams
  VerifyReq* vreq;                 // deferred verification requests
  unsigned long long* vcount;      // their count (may exceed vcap)
  int64_t vcap;
  unsigned long long* tmargin;     // largest drift margin of a trusted FP32 value (float bits)
  unsigned long long* overflow;    // candidates verified in place (request buffer full)
  // MATRIX_SUMMARY: the grid and its geometry (JoinParams), the current
  // problem's targets
  int knn_k;  // APPROX_ALL_NEIGHBORS: list length (0 otherwise)
  unsigned* mat;
  int64_t mat_w, mat_h;
  int64_t rpc, cpc;
  uint64_t rpc_magic, cpc_magic;
  bool mcol, mrow;
  // exact form: verification requests of the current unit, and whether it
  // is left to the FP64 band kernel (more than the budget, or the buffer full)
  unsigned unit_reqs;
  unsigned unit_wide;   // those whose bound exceeds kWideBound
  unsigned unit_lost;
  unsigned budget, wide_budget;
};

struct Smem {
  union {
    struct {
      // {df.x, df.y} and {dg.x, dg.y} per staged column pair: separate
      // 8-byte arrays, so that 64-bit loads at a stride of 9 slots meet no
      // bank conflict
      float2 c_df[kPadG];
      float2 c_dg[kPadG];
      float2 c_iv[kPadG];  // {inv.x, inv.y}
    } s;
    struct {
      float2 xr[kAnchorChunk];    // centred row windows of both segments (chunk)
      float2 yc[kYPad];           // column samples (block-relative), padded
      union {
        float2 cb[2][kSpanBlk];   // {bhi, blo} of the blocks of the staged span
        double cbd[2][kSpanBlk];  // exact form: the block offsets in FP64
      };
    } a;
  } u;
  float2 c_best[kCols + kCols / 8];  // at padc(ring column), as c_df
  // per 8-column ring block (entry kBlocks repeats block 0): smallest best,
  // largest inverse norm, largest |df|, |dg|
  float2 c_blkmin[kBlocks + 1];
  float2 c_blkmax_iv[kBlocks + 1];
  float4 c_blkmax_fg[kBlocks + 1];
  float4 r_fg[kSlab];
  float2 r_iv[kSlab];
  float2 r_best[kSlab];
  float2 r_stepmin[kSteps];
  float2 r_stepmax_iv[kSteps];
  float4 r_stepmax_fg[kSteps];
  SlowItem queue[kWarps][kQueue];
  Problem prob;  // the current unit's band problem
  long long unit, band, unit_in_band;
  int prob_index;
  SlowCtx cx;
  // each warp's block of the request buffer and its used slots
  unsigned long long rq_base[kWarps];
  int rq_used[kWarps];
};

// Filter-table entry: smallest best, largest inverse norm, largest |df|,
// |dg| (per segment), over a set of columns or rows.
struct TableEntry {
  float2 mn, mx;
  float4 mf;
};

// One column's or row's entry; a NaN inverse norm (window that cannot match)
// counts as 0, as fmaxf against a 0 start would.
__device__ __forceinline__ TableEntry table_entry(float4 f, float2 iv, float2 best) {
  TableEntry e;
  e.mn = best;
  e.mx = make_float2(fmaxf(0.f, iv.x), fmaxf(0.f, iv.y));
  e.mf = make_float4(fabsf(f.x), fabsf(f.y), fabsf(f.z), fabsf(f.w));
  return e;
}

// Exact form: dg = (b - mu') + (a - mu) is a rounded sum, off by up to 2^-52
// of its terms (|dg| + 3 |df| bounds them), which a cancelled |dg| would not
// show; 2^-20 |df| in its place keeps the step's bound above that.
__device__ __forceinline__ void floor_dg(TableEntry& e) {
  e.mf.z = fmaxf(e.mf.z, 9.6e-7f * e.mf.x);
  e.mf.w = fmaxf(e.mf.w, 9.6e-7f * e.mf.y);
}

__device__ __forceinline__ void combine(TableEntry& a, const TableEntry& b) {
  a.mn = make_float2(fminf(a.mn.x, b.mn.x), fminf(a.mn.y, b.mn.y));
  a.mx = make_float2(fmaxf(a.mx.x, b.mx.x), fmaxf(a.mx.y, b.mx.y));
  a.mf = make_float4(fmaxf(a.mf.x, b.mf.x), fmaxf(a.mf.y, b.mf.y),
                     fmaxf(a.mf.z, b.mf.z), fmaxf(a.mf.w, b.mf.w));
}

// Reduces an entry over aligned groups of 8 lanes (whole warp active).
__device__ __forceinline__ void reduce8(TableEntry& e) {
#pragma unroll
  for (int o = 1; o < 8; o <<= 1) {
    TableEntry x;
    x.mn.x = __shfl_xor_sync(0xffffffffu, e.mn.x, o);
    x.mn.y = __shfl_xor_sync(0xffffffffu, e.mn.y, o);
    x.mx.x = __shfl_xor_sync(0xffffffffu, e.mx.x, o);
    x.mx.y = __shfl_xor_sync(0xffffffffu, e.mx.y, o);
    x.mf.x = __shfl_xor_sync(0xffffffffu, e.mf.x, o);
    x.mf.y = __shfl_xor_sync(0xffffffffu, e.mf.y, o);
    x.mf.z = __shfl_xor_sync(0xffffffffu, e.mf.z, o);
    x.mf.w = __shfl_xor_sync(0xffffffffu, e.mf.w, o);
    combine(e, x);
  }
}

template <int P>
struct Parity {
  static constexpr int value = P;
};

static_assert(kSlab == kThreads, "one staged row per thread");
static_assert(kCols % kThreads == 0, "whole warps stage the columns");

// Four CTAs per SM: 4 x (shared memory + 1 KB reserved) within 228 KB.
static_assert(sizeof(Smem) + 1024 <= 228 * 1024 / 4, "shared memory exceeds 4 CTAs/SM");

__device__ __forceinline__ int padc(int c) { return c + (c >> 3); }
// Ring column of slab-relative column c (0 <= c < kCols).
__device__ __forceinline__ int ringc(int ring0, int c) {
  const int r = ring0 + c;
  return r >= kCols ? r - kCols : r;
}

// {df.x, df.y, dg.x, dg.y} of the staged column in padded slot `slot`.
__device__ __forceinline__ float4 col_fg(const Smem& sm, int slot) {
  const float2 a = sm.u.s.c_df[slot], b = sm.u.s.c_dg[slot];
  return make_float4(a.x, a.y, b.x, b.y);
}
__device__ __forceinline__ int pady2(int x) { return x + (x >> 3) * 2; }

// Offset of block b relative to block b0, as the float sum of the two
// blocks' hi/lo parts: exact while the two offsets are within a factor of two.
__device__ __forceinline__ float block_delta(const SeriesDev& S, int64_t b, int64_t b0) {
  return (S.bhi[b] - S.bhi[b0]) + (S.blo[b] - S.blo[b0]);
}

// Partial covariance of row window i and column window j over the terms
// t in [tb, te), FP32: each factor formed as (sample relative to its block
// offset) + (block offset - window mean), summed per run of terms that share
// both blocks.
__device__ __forceinline__ float cov_part(const SeriesDev& R, const SeriesDev& C,
                                          int64_t i, int64_t j, int64_t tb, int64_t te_all) {
  const int sh = R.bshift;
  const int64_t bi = i >> sh, bj = j >> sh;
  const float mri = R.mu_rel[i], mcj = C.mu_rel[j];
  float acc = 0.f;
  int64_t t = tb;
  while (t < te_all) {
    const int64_t br = (i + t) >> sh, bc = (j + t) >> sh;
    int64_t te = ((br + 1) << sh) - i;
    const int64_t te2 = ((bc + 1) << sh) - j;
    if (te2 < te) te = te2;
    if (te_all < te) te = te_all;
    const float xc = block_delta(R, br, bi) - mri;
    const float yc = block_delta(C, bc, bj) - mcj;
    float p0 = 0.f, p1 = 0.f, p2 = 0.f, p3 = 0.f;
    int64_t u = t;
    for (; u + 3 < te; u += 4) {
      p0 = fmaf(R.T32[i + u] + xc, C.T32[j + u] + yc, p0);
      p1 = fmaf(R.T32[i + u + 1] + xc, C.T32[j + u + 1] + yc, p1);
      p2 = fmaf(R.T32[i + u + 2] + xc, C.T32[j + u + 2] + yc, p2);
      p3 = fmaf(R.T32[i + u + 3] + xc, C.T32[j + u + 3] + yc, p3);
    }
    for (; u < te; ++u) p0 = fmaf(R.T32[i + u] + xc, C.T32[j + u] + yc, p0);
    acc += (p0 + p1) + (p2 + p3);
    t = te;
  }
  return acc;
}

// The same covariance computed by a whole warp: lane l sums the terms
// t = l, l + 32, ...; the partial sums meet in a shuffle reduction.  The
// samples' centring terms belong to their blocks, of which a window touches
// 18 at most (block_shift()): each lane forms one block's, and a sample's
// comes by a shuffle (loaded and formed again for every sample, the seeds of
// 2^20 windows of m = 1024 took 2.19 ms, now 0.89: 9.3 TB/s from L2).
__device__ __forceinline__ float verify_cov_warp(const SeriesDev& R, const SeriesDev& C,
                                                 int64_t i, int64_t j, int64_t m, int lane) {
  const int sh = R.bshift, mi = static_cast<int>(m);
  const int64_t bi = i >> sh, bj = j >> sh;
  const float mri = R.mu_rel[i], mcj = C.mu_rel[j];
  // windows start oi, oj samples into their blocks
  const int oi = static_cast<int>(i - (bi << sh)), oj = static_cast<int>(j - (bj << sh));
  const int br = lane < ((oi + mi - 1) >> sh) + 1 ? lane : 0;
  const int bc = lane < ((oj + mi - 1) >> sh) + 1 ? lane : 0;
  const float xb = ((R.bhi[bi + br] - R.bhi[bi]) + (R.blo[bi + br] - R.blo[bi])) - mri;
  const float yb = ((C.bhi[bj + bc] - C.bhi[bj]) + (C.blo[bj + bc] - C.blo[bj])) - mcj;
  const float* __restrict__ tr = R.T32 + i;
  const float* __restrict__ tc = C.T32 + j;
  float acc[4] = {0.f, 0.f, 0.f, 0.f};
  for (int t0 = lane; t0 - lane < mi; t0 += 128) {
    float x[4], y[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const int t = t0 + 32 * u;
      x[u] = t < mi ? tr[t] : 0.f;
      y[u] = t < mi ? tc[t] : 0.f;
    }
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const int t = t0 + 32 * u;
      const float dx = __shfl_sync(0xffffffffu, xb, (oi + t) >> sh);
      const float dy = __shfl_sync(0xffffffffu, yb, (oj + t) >> sh);
      if (t < mi) acc[u] = fmaf(x[u] + dx, y[u] + dy, acc[u]);
    }
  }
  float a = (acc[0] + acc[1]) + (acc[2] + acc[3]);
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) a += __shfl_xor_sync(0xffffffffu, a, o);
  return a;
}

// The whole covariance, one lane (the diagonal seeds).
__device__ __noinline__ float verify_cov_lane(const SeriesDev& R, const SeriesDev& C,
                                              int64_t i, int64_t j, int64_t m) {
  return cov_part(R, C, i, j, 0, m);
}


__device__ __forceinline__ void publish(Smem& sm, const SlowCtx& cx, float rv, int64_t i,
                                        int64_t j, int rslot, int cslot, int g) {
  const float rb = g ? sm.r_best[rslot].y : sm.r_best[rslot].x;
  const float cb = g ? sm.c_best[padc(cslot)].y : sm.c_best[padc(cslot)].x;
  if (rv > rb) {
    atomicMax(reinterpret_cast<u64*>(cx.key_row + i),
              make_key(q_from_float_bits(__float_as_uint(rv), cx.kl.frac_bits), j, cx.kl));
    // The float copies only filter candidates; a racing store of a smaller
    // value costs extra work later, never a wrong result.
    if (g) sm.r_best[rslot].y = rv; else sm.r_best[rslot].x = rv;
  }
  if (rv > cb) {
    atomicMax(reinterpret_cast<u64*>(cx.key_col + j),
              make_key(q_from_float_bits(__float_as_uint(rv), cx.kl.frac_bits), i, cx.kl));
    if (g) sm.c_best[padc(cslot)].y = rv; else sm.c_best[padc(cslot)].x = rv;
  }
}

// A list's filter value: its k-th best (rounded down), at least the threshold.
__device__ __forceinline__ float knn_floor(const uint64_t* list, int k, float thr,
                                           const KeyLayout& kl) {
  return fmaxf(key_corr_floor(list[k - 1], kl), thr);
}

// APPROX_ALL_NEIGHBORS counterpart of publish(): a cell above its row's
// (column's) k-th best enters that window's list; the shared filter value
// then follows the list's new k-th entry.
__device__ __noinline__ void knn_publish(Smem& sm, const SlowCtx& cx, float rv, int64_t i,
                                         int64_t j, int rslot, int cslot, int g) {
  if (!(rv > cx.thr)) return;
  const Problem& pr = *cx.pr;
  const int k = cx.knn_k;
  const float rb = g ? sm.r_best[rslot].y : sm.r_best[rslot].x;
  const float cb = g ? sm.c_best[padc(cslot)].y : sm.c_best[padc(cslot)].x;
  const uint64_t q = q_from_float_bits(__float_as_uint(rv), cx.kl.frac_bits);
  if (rv > rb && pr.key_row) {
    u64* list = reinterpret_cast<u64*>(pr.key_row + i * k);
    topk_insert(list, k, make_key(q, j, cx.kl));
    const float nb = knn_floor(pr.key_row + i * k, k, cx.thr, cx.kl);
    if (g) sm.r_best[rslot].y = nb; else sm.r_best[rslot].x = nb;
  }
  if (rv > cb && pr.key_col) {
    u64* list = reinterpret_cast<u64*>(pr.key_col + j * k);
    topk_insert(list, k, make_key(q, i, cx.kl));
    const float nb = knn_floor(pr.key_col + j * k, k, cx.thr, cx.kl);
    if (g) sm.c_best[padc(cslot)].y = nb; else sm.c_best[padc(cslot)].x = nb;
  }
}

// One cell of the exact path: publish (or add) its FP32 value when that is
// safe, else queue a verification request at `slot`.
__device__ __forceinline__ void exact_cell(Smem& sm, const SlowCtx& cx, float rv, float mk,
                                           bool cand, bool req, unsigned long long slot,
                                           int64_t i, int64_t j, int rslot, int cslot, int g,
                                           float& add, float& tmax, int& nreq) {
  if (!cand) return;
  if (req) {
    ++nreq;
    if (slot < static_cast<unsigned long long>(cx.vcap)) {
      // (1NN: the lower bound raises the filters at once; a k-best list
      // would keep it beside the verified value)
      if (!cx.sum_mode && !cx.knn_k) publish(sm, cx, rv - mk, i, j, rslot, cslot, g);
      VerifyReq q;
      q.i = static_cast<uint64_t>(i) | (static_cast<uint64_t>(cx.prob) << 40);
      q.d = static_cast<uint32_t>(j - i);
      q.ub = rv + mk;
      cx.vreq[slot] = q;
    } else {
      // request buffer full: verified in place by this lane (slow: the
      // counted overflow makes later joins size the buffer for it)
      const Problem& pr = *cx.pr;
      // (the dot inline: a call from here makes every band kernel that
      // calls the exact path keep more registers live across it)
      const float ev = (cov_part(pr.R, pr.C, i, j, 0, cx.m) * pr.C.inv32[j]) * pr.R.inv32[i];
      atomicAdd(cx.overflow, 1ull);
      if (cx.sum_mode) add = ev > cx.thr ? ev : 0.f;
      else if (cx.knn_k) knn_publish(sm, cx, ev, i, j, rslot, cslot, g);
      else publish(sm, cx, ev, i, j, rslot, cslot, g);
    }
  } else if (cx.sum_mode) {
    add = rv > cx.thr ? rv : 0.f;
    if (add != 0.f) tmax = fmaxf(tmax, mk);
  } else {
    if (cx.knn_k) knn_publish(sm, cx, rv, i, j, rslot, cslot, g);
    else publish(sm, cx, rv, i, j, rslot, cslot, g);
    tmax = fmaxf(tmax, mk);
  }
}

// The unused slots of the warp's block of the request buffer
// become requests that rule themselves out.
__device__ __forceinline__ void close_requests(Smem& sm, const SlowCtx& cx, int warp, int lane) {
  const unsigned long long base = sm.rq_base[warp];
  for (int s = sm.rq_used[warp] + lane; s < kReqChunk; s += 32)
    if (base + s < static_cast<unsigned long long>(cx.vcap)) cx.vreq[base + s] = VerifyReq{0, 0, -4.f};
}

// n consecutive slots of the request buffer for the warp, from a block of
// kReqChunk that it takes at a time, so that the global counter's round trip
// is paid once per block and not once per row of candidates.  Called by the
// whole warp; more than a block's slots come as whole blocks.
__device__ __forceinline__ unsigned long long take_requests(Smem& sm, const SlowCtx& cx, int warp,
                                                            int lane, int n) {
  int used = sm.rq_used[warp];
  unsigned long long base = sm.rq_base[warp];
  if (used + n > kReqChunk) {
    close_requests(sm, cx, warp, lane);
    const int whole = (n - 1) / kReqChunk * kReqChunk;  // slots before the last block
    if (lane == 0) base = atomicAdd(cx.vcount, static_cast<unsigned long long>(whole + kReqChunk));
    base = __shfl_sync(0xffffffffu, base, 0) + whole;
    used = -whole;
  }
  __syncwarp();
  if (lane == 0) {
    sm.rq_base[warp] = base;
    sm.rq_used[warp] = used + n;
  }
  __syncwarp();
  return base + used;
}

// Sum of v over the lanes up to this one.
__device__ __forceinline__ int warp_prefix(int v, int lane) {
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int w = __shfl_up_sync(0xffffffffu, v, o);
    if (lane >= o) v += w;
  }
  return v;
}

// Exact path of queued blocks, 8 lanes per block (four blocks per pass):
// lane k holds the covariances of diagonal k in both segments (an f32x2
// pair, as the fast path holds them) at the block's end and visits the
// block's rows (8 per step), each with the covariance the fast path used
// there.  kMerged (the per-cell-filter kernels): one pass, rows last to
// first, stepping the covariance back over each row before checking it.
// Otherwise (the per-step-bound kernels) the covariance is first rewound to
// the block's start, then the rows are checked first to last (measured: the
// one-pass form is 6-7% faster on the AB and batched joins of short windows,
// 1.3% slower on the self-join of 1024-sample windows).  Every cell that may
// improve its row or column is published with its FP32 value when its
// margin is within kTrust.  A cell with a larger margin is published with the lower bound
// rv - margin (so the filters rise at once) and appended to the
// verification requests, which verify_requests_kernel settles after the
// join.  Returns the lane's number of requests.
template <bool kMerged>
__device__ __noinline__ int drain_queue(Smem& sm, int warp, int count, int lane) {
  __syncwarp();  // the queue was written by other lanes
  const SlowCtx& cx = sm.cx;
  const int k = lane & 7;
  int nreq = 0;
  float tmax = 0.f;  // largest margin of a value published or added unverified
  for (int p = 0; p < count; p += 4) {
    // every lane runs the pass (warp-wide request reservation); a lane
    // without a block carries the first queued one and checks nothing
    const int item = p + (lane >> 3);
    const bool act = item < count;
    const SlowItem& it = sm.queue[warp][act ? item : 0];
    float2 c = it.cov[k];
    const float2 vw = it.vw;
    const int s0 = it.s & 255;
    const int nrows = act ? kRows * ((it.s >> 8) & 255) : 0;
    const int msk = (it.s >> 16) & 15;  // segments to walk, per step of the block
    // the blocks of a pass may differ in length: the row loop below runs
    // the longest on every lane (its ballots need the whole warp)
    const int nrows_w = static_cast<int>(__reduce_max_sync(0xffffffffu, static_cast<unsigned>(nrows)));
    const int r0 = s0 * kRows;
    const int cb0 = 8 * (s0 + it.owner) + k;  // staged column at row 0
    if constexpr (!kMerged) {
#pragma unroll 8
      for (int rr = nrows - 1; rr >= 0; --rr) {
        const float4 rf = sm.r_fg[r0 + rr];
        const float4 cf = col_fg(sm, padc(ringc(cx.ring0, cb0 + rr)));
        c = fma2(make_float2(-rf.x, -rf.y), make_float2(cf.z, cf.w), c);
        c = fma2(make_float2(-cf.x, -cf.y), make_float2(rf.z, rf.w), c);
      }
    }
    const float2 vk = make_float2(kBoundC * kEps * sqrtf(kRows * vw.x),
                                  kBoundC * kEps * sqrtf(kRows * vw.y));
    const int64_t jd = cx.D0 + it.owner * kDiags + k;  // the lane's diagonal
    // kMerged, rows last to first: stepping back over row rr leaves c at the
    // covariance the fast path used in row rr.  The rows' order and timing
    // show where two cells have equal FP32 values, of which the first one
    // published stays the partner: filtering a step's rows together before
    // settling them made the m = 1024 form 5% faster (2^20 windows, band
    // kernel 94.7 -> 90.0 ms) and named another partner for one window in
    // ten million; so did `>=` in publish(), for two in a million.
#pragma unroll 1
    for (int rw = kMerged ? nrows_w - 1 : 0; kMerged ? rw >= 0 : rw < nrows_w;
         rw += kMerged ? -1 : 1) {
      const bool live = rw < nrows;
      const int rr = live ? rw : 0;  // rows past the block's end read row 0
      const int cs = cb0 + rr;
      const int rcs = ringc(cx.ring0, cs);  // its ring column
      const float4 rf = sm.r_fg[r0 + rr];
      const float4 cf = col_fg(sm, padc(rcs));
      if constexpr (kMerged) {
        if (live) {
          c = fma2(make_float2(-rf.x, -rf.y), make_float2(cf.z, cf.w), c);
          c = fma2(make_float2(-cf.x, -cf.y), make_float2(rf.z, rf.w), c);
        }
      }
      const float2 ivr = sm.r_iv[r0 + rr];
      const float2 ivc = sm.u.s.c_iv[padc(rcs)];
      const float2 rv = mul2(mul2(c, ivc), ivr);  // the fast path's rounding
      const float2 mk = mul2(mul2(vk, ivc), ivr);
      const float2 rb = sm.r_best[r0 + rr];
      const float2 cbv = sm.c_best[padc(rcs)];
      // the value to beat: the row's and column's bests, or the threshold
      const float tx = cx.sum_mode ? cx.thr : fminf(rb.x, cbv.x);
      const float ty = cx.sum_mode ? cx.thr : fminf(rb.y, cbv.y);
      const int sm2 = msk >> (2 * (rw >> 3));
      const bool cx_ = live && (sm2 & 1) && rv.x + mk.x > tx;
      const bool cy_ = live && (sm2 & 2) && rv.y + mk.y > ty;
      // SUM_THRESH: a cell surely above the threshold counts with its FP32 r
      const bool qx = cx_ && mk.x > kTrust && !(cx.sum_mode && rv.x - mk.x > tx);
      const bool qy = cy_ && mk.y > kTrust && !(cx.sum_mode && rv.y - mk.y > ty);
      const unsigned mx = __ballot_sync(0xffffffffu, qx), my = __ballot_sync(0xffffffffu, qy);
      unsigned long long sx = 0, sy = 0;
      if (mx | my) {
        const unsigned long long base = take_requests(sm, cx, warp, lane, __popc(mx) + __popc(my));
        const unsigned lt = (1u << lane) - 1u;
        sx = base + __popc(mx & lt) + __popc(my & lt);
        sy = sx + (qx ? 1u : 0u);
      }
      float ax = 0.f, ay = 0.f;  // SUM_THRESH: what the cells add to their rows and column
      if (cx_ || cy_) {
        const int64_t i0 = cx.rbase[0] + r0 + rr, i1 = cx.rbase[1] + r0 + rr;
        exact_cell(sm, cx, rv.x, mk.x, cx_, qx, sx, i0, i0 + jd, r0 + rr, rcs, 0, ax, tmax, nreq);
        exact_cell(sm, cx, rv.y, mk.y, cy_, qy, sy, i1, i1 + jd, r0 + rr, rcs, 1, ay, tmax, nreq);
      }
      if (cx.sum_mode) {
        // the 8 diagonals of a block meet in one row: reduce over its lanes
        // (k = lane bits 0-2) before the shared-memory atomics
        if (ax != 0.f) atomicAdd(&sm.c_best[padc(rcs)].x, ax);
        if (ay != 0.f) atomicAdd(&sm.c_best[padc(rcs)].y, ay);
        float2 rs = make_float2(ax, ay);
#pragma unroll
        for (int o = 1; o < 8; o <<= 1) {
          rs.x += __shfl_xor_sync(0xffffffffu, rs.x, o);
          rs.y += __shfl_xor_sync(0xffffffffu, rs.y, o);
        }
        if (k == 0) {
          if (rs.x != 0.f) atomicAdd(&sm.r_best[r0 + rr].x, rs.x);
          if (rs.y != 0.f) atomicAdd(&sm.r_best[r0 + rr].y, rs.y);
        }
      }
      if constexpr (!kMerged) {
        c = fma2(make_float2(cf.x, cf.y), make_float2(rf.z, rf.w), c);
        c = fma2(make_float2(rf.x, rf.y), make_float2(cf.z, cf.w), c);
      }
    }
  }
  // the trusted margins, one atomic per drain (non-negative floats order as
  // their bit patterns)
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) tmax = fmaxf(tmax, __shfl_xor_sync(0xffffffffu, tmax, o));
  if (lane == 0 && tmax > 0.f) atomicMax(cx.tmargin, static_cast<unsigned long long>(__float_as_uint(tmax)));
  __syncwarp();
  return nreq;
}

// Exact form: counts n requests, `wide` of them of wide bounds and the last
// below slot `end`, against what the unit may make.
__device__ __forceinline__ void spend_requests(Smem& sm, const SlowCtx& cx, unsigned n,
                                               unsigned wide, unsigned long long end) {
  if (atomicAdd(&sm.cx.unit_reqs, n) + n > cx.budget ||
      (wide && atomicAdd(&sm.cx.unit_wide, wide) + wide > cx.wide_budget) ||
      end > static_cast<unsigned long long>(cx.vcap))
    sm.cx.unit_lost = 1;
}

// Exact form: writes the requests of the lanes that qx, qy mark (segments x
// and y of cells (i, i + d)).  Called by the whole warp; returns the number
// written.
__device__ __forceinline__ int push_requests(Smem& sm, const SlowCtx& cx, int warp, int lane,
                                             bool qx, bool qy, float2 rv, float2 mk, int64_t ix,
                                             int64_t iy, int64_t d) {
  const unsigned mx = __ballot_sync(0xffffffffu, qx), my = __ballot_sync(0xffffffffu, qy);
  const int n = __popc(mx) + __popc(my);
  if (n == 0) return 0;
  const unsigned long long base = take_requests(sm, cx, warp, lane, n);
  const unsigned lt = (1u << lane) - 1u;
  VerifyReq rq;
  rq.d = static_cast<uint32_t>(d);
  const unsigned long long sx = base + __popc(mx & lt);
  const unsigned long long sy = base + __popc(mx) + __popc(my & lt);
  if (qx && sx < static_cast<unsigned long long>(cx.vcap)) {
    rq.i = static_cast<uint64_t>(ix) | (static_cast<uint64_t>(cx.prob) << 40);
    rq.ub = rv.x + mk.x;
    cx.vreq[sx] = rq;
  }
  if (qy && sy < static_cast<unsigned long long>(cx.vcap)) {
    rq.i = static_cast<uint64_t>(iy) | (static_cast<uint64_t>(cx.prob) << 40);
    rq.ub = rv.y + mk.y;
    cx.vreq[sy] = rq;
  }
  const unsigned wide = __popc(__ballot_sync(0xffffffffu, qx && mk.x > kWideBound)) +
                        __popc(__ballot_sync(0xffffffffu, qy && mk.y > kWideBound));
  if (lane == 0) spend_requests(sm, cx, static_cast<unsigned>(n), wide, base + n);
  __syncwarp();
  return n;
}

// Exact form: a candidate's lower bound lb raises its row's and its column's
// best at once, in the keys and in the staged copies (which only filter: a
// racing store of a smaller value costs extra work, never a wrong result).
__device__ __forceinline__ void publish_bound(Smem& sm, const SlowCtx& cx, float lb, int64_t i,
                                              int64_t j, int rslot, int cslot, int g) {
  if (!(lb > -2.f)) return;
  float& rb = g ? sm.r_best[rslot].y : sm.r_best[rslot].x;
  float& cb = g ? sm.c_best[padc(cslot)].y : sm.c_best[padc(cslot)].x;
  const uint64_t q = q_from_float_bits(__float_as_uint(lb), cx.kl.frac_bits);
  if (lb > rb) {
    atomicMax(reinterpret_cast<u64*>(cx.key_row + i), make_key(q, j, cx.kl));
    rb = lb;
  }
  if (lb > cb) {
    atomicMax(reinterpret_cast<u64*>(cx.key_col + j), make_key(q, i, cx.kl));
    cb = lb;
  }
}

// Exact matrix form: the smallest bound of the grid entries that the windows
// a .. a + da (grid rows) and b .. b + db (grid columns) fall in; the spans are
// shorter than an entry's, so that is two entries each way at most.
__device__ __forceinline__ float mat_block_floor(const SlowCtx& cx, int64_t a, int64_t da,
                                                 int64_t b, int64_t db) {
  const int64_t qa = div_magic(a, cx.rpc_magic), qb = div_magic(b, cx.cpc_magic);
  const bool ra = a - qa * cx.rpc + da >= cx.rpc && qa + 1 < cx.mat_h;
  const bool rb = b - qb * cx.cpc + db >= cx.cpc && qb + 1 < cx.mat_w;
  const unsigned* e = cx.mat + qa * cx.mat_w + qb;
  unsigned lo = e[0];
  if (ra) lo = min(lo, e[cx.mat_w]);
  if (rb) lo = min(lo, e[1]);
  if (ra && rb) lo = min(lo, e[cx.mat_w + 1]);
  return lo ? float_of_ord(lo) : -3.f;
}
__device__ __forceinline__ float mat_cell_floor(const SlowCtx& cx, int64_t i, int64_t j) {
  float lo = kNoTarget;
  if (cx.mcol) lo = mat_block_floor(cx, i, 0, j, 0);
  if (cx.mrow) lo = fminf(lo, mat_block_floor(cx, j, 0, i, 0));
  return lo;
}

// drain_queue() of the exact form: the same walk (rows last to first, the
// covariance stepped back over each row), with the deterministic bound.  An
// item's vw is E at the block's end plus the block's own roundings again,
// for the steps back.
template <bool kMat>
__device__ __noinline__ int drain_exact(Smem& sm, int warp, int count, int lane) {
  __syncwarp();  // the queue was written by other lanes
  // (in registers: read again after every store otherwise; m = 1024 with gaps
  // 2.89 -> 2.75 ms.  The mixed form's exact path has no registers left for
  // it: its kernels spilled, 9% slower.)
  const SlowCtx cx = sm.cx;
  const int k = lane & 7;
  int nreq = 0;
  for (int p = 0; p < count; p += 4) {
    // a unit left to the FP64 kernel needs no more requests (lane 0's view:
    // another warp may be setting it)
    if (__shfl_sync(0xffffffffu, *const_cast<volatile unsigned*>(&sm.cx.unit_lost), 0)) break;
    const int item = p + (lane >> 3);
    const bool act = item < count;
    const SlowItem& it = sm.queue[warp][act ? item : 0];
    float2 c = it.cov[k];
    const float2 vw = make_float2(kBoundSlack * it.vw.x, kBoundSlack * it.vw.y);
    const int s0 = it.s & 255;
    const int nrows = act ? kRows * ((it.s >> 8) & 255) : 0;
    const int nrows_w = static_cast<int>(__reduce_max_sync(0xffffffffu, static_cast<unsigned>(nrows)));
    const int r0 = s0 * kRows;
    const int cb0 = 8 * (s0 + it.owner) + k;           // staged column at row 0
    const int64_t jd = cx.D0 + it.owner * kDiags + k;  // the lane's diagonal
    if constexpr (!kMat) {
      // A step's rows are first all filtered, their loads in flight together;
      // then one reservation holds every candidate's request, and each lane
      // writes and publishes its own (those that the bests raised meanwhile
      // rule out as requests that rule themselves out).  Row by row, a row
      // with candidates was ~1300 cycles of one warp's latency: band kernels
      // and verification of 40009 samples with gaps, m = 1024, 2.87 -> 2.52 ms,
      // 60000 x 30011, m = 256, 1.25 -> 1.16, 1000, m = 50, 0.130 -> 0.118.
#pragma unroll 1
      for (int b = nrows_w / kRows - 1; b >= 0; --b) {
        const bool live = b * kRows < nrows;
        const int q0 = live ? b * kRows : 0;  // a step past the block's end reads its first
        float2 rvs[kRows];
        unsigned cand = 0;  // bit u: row u of the first segment, bit u + 8: of the second
#pragma unroll
        for (int u = kRows - 1; u >= 0; --u) {
          const int rr = q0 + u;
          const int slot = padc(ringc(cx.ring0, cb0 + rr));
          const float4 rf = sm.r_fg[r0 + rr];
          const float4 cf = col_fg(sm, slot);
          if (live) {
            c = fma2(make_float2(-rf.x, -rf.y), make_float2(cf.z, cf.w), c);
            c = fma2(make_float2(-cf.x, -cf.y), make_float2(rf.z, rf.w), c);
          }
          const float2 ivr = sm.r_iv[r0 + rr];
          const float2 ivc = sm.u.s.c_iv[slot];
          const float2 rv = mul2(mul2(c, ivc), ivr);
          const float2 mk = mul2(mul2(vw, ivc), ivr);
          const float2 rb = sm.r_best[r0 + rr];
          const float2 cbv = sm.c_best[slot];
          // (false for NaN: excluded diagonals, windows that cannot match)
          if (rv.x + (mk.x + kAbsSlack) > fminf(rb.x, cbv.x)) cand |= 1u << u;
          if (rv.y + (mk.y + kAbsSlack) > fminf(rb.y, cbv.y)) cand |= 256u << u;
          rvs[u] = rv;
        }
        if (!live) cand = 0;
        const int mine = __popc(cand);
        const int upto = warp_prefix(mine, lane);
        const int total = __shfl_sync(0xffffffffu, upto, 31);
        if (total == 0) continue;
        const unsigned long long base = take_requests(sm, cx, warp, lane, total);
        unsigned long long slot = base + (upto - mine);
        unsigned real = 0, wide = 0;
#pragma unroll 1
        while (cand) {
          const int bit = 31 - __clz(cand);
          cand &= ~(1u << bit);
          const int u = bit & 7, g = bit >> 3, rr = q0 + u;
          const int rcs = ringc(cx.ring0, cb0 + rr);
          const float2 mk2 = mul2(mul2(vw, sm.u.s.c_iv[padc(rcs)]), sm.r_iv[r0 + rr]);
          const float2 rb = sm.r_best[r0 + rr];
          const float2 cbv = sm.c_best[padc(rcs)];
          const float rv = g ? rvs[u].y : rvs[u].x, mk = (g ? mk2.y : mk2.x) + kAbsSlack;
          const bool ok = rv + mk > (g ? fminf(rb.y, cbv.y) : fminf(rb.x, cbv.x));
          const int64_t i = cx.rbase[g] + r0 + rr;
          if (slot < static_cast<unsigned long long>(cx.vcap)) {
            VerifyReq rq;
            rq.i = static_cast<uint64_t>(i) | (static_cast<uint64_t>(cx.prob) << 40);
            rq.d = static_cast<uint32_t>(jd);
            rq.ub = ok ? rv + mk : -4.f;
            cx.vreq[slot] = rq;
          }
          ++slot;
          if (!ok) continue;
          ++real;
          wide += mk > kWideBound ? 1u : 0u;
          // (one cell's bound says nothing of a window's k-th best)
          if (!cx.knn_k) publish_bound(sm, cx, rv - mk, i, i + jd, r0 + rr, rcs, g);
        }
        __syncwarp();
        real = __reduce_add_sync(0xffffffffu, real);
        wide = __reduce_add_sync(0xffffffffu, wide);
        nreq += static_cast<int>(real);
        if (lane == 0) spend_requests(sm, cx, real, wide, base + total);
      }
    } else {
      // matrix: most rows hold a candidate of some grid entry's floor test
#pragma unroll 1
      for (int rw = nrows_w - 1; rw >= 0; --rw) {
        const bool live = rw < nrows;
        const int rr = live ? rw : 0;  // rows past the block's end read row 0
        const int slot = padc(ringc(cx.ring0, cb0 + rr));
        const float4 rf = sm.r_fg[r0 + rr];
        const float4 cf = col_fg(sm, slot);
        if (live) {
          c = fma2(make_float2(-rf.x, -rf.y), make_float2(cf.z, cf.w), c);
          c = fma2(make_float2(-cf.x, -cf.y), make_float2(rf.z, rf.w), c);
        }
        const float2 ivr = sm.r_iv[r0 + rr];
        const float2 ivc = sm.u.s.c_iv[slot];
        const float2 rv = mul2(mul2(c, ivc), ivr);
        const float2 mk0 = mul2(mul2(vw, ivc), ivr);
        const float2 mk = make_float2(mk0.x + kAbsSlack, mk0.y + kAbsSlack);
        const int64_t i0 = cx.rbase[0] + r0 + rr, i1 = cx.rbase[1] + r0 + rr;
        // (false for NaN: excluded diagonals, windows that cannot match)
        bool cx_ = live && rv.x + mk.x > cx.thr, cy_ = live && rv.y + mk.y > cx.thr;
        if (cx_) cx_ = rv.x + mk.x > mat_cell_floor(cx, i0, i0 + jd);
        if (cy_) cy_ = rv.y + mk.y > mat_cell_floor(cx, i1, i1 + jd);
        nreq += push_requests(sm, cx, warp, lane, cx_, cy_, rv, mk, i0, i1, jd);
      }
    }
  }
  __syncwarp();
  return lane == 0 ? nreq : 0;
}

// Bound on the error of a thread's FP32 anchors (exact form), per segment,
// from the squared norms of what it multiplied: x2 of the row window
// (centred in FP64, rounded once), y2 the sum of T32^2 + d^2 over the column
// samples y = T32 + d it read (T32 and d rounded once each, so that
// ||(|T32| + |d| + |y|)|| <= sqrt(8 y2)), and the largest mean difference ek
// between its windows.  Runs of 32 products, ceil(m / 32) sums of runs and
// the correction ek * sum x; with ||y|| <= sqrt(8 y2) / 2,
//   E <= u ||x|| ((35 + m/32) / 2 + 2) sqrt(8 y2) + (38 + m/32) ek sqrt(m))
// (inputs 1.5 u ||x|| sqrt(8 y2), the rest accumulation).
__device__ __forceinline__ float anchor_bound(float x2, float y2, float ek, float m) {
  const float runs = m * (1.f / 32.f);
  return kBoundSlack * kBoundSlack * kEps * sqrtf(x2) *
         ((0.5f * (35.f + runs) + 2.f) * sqrtf(8.f * y2) + (38.f + runs) * ek * sqrtf(m));
}

// SUM_THRESH: the cells of a thread-step that lie within the step's margin
// m of the threshold (flags fx, fy per segment; rare), walked again by their
// lane alone from the step's start (rewound from the covariances at its
// end, as the exact path rewinds).  Each such cell is decided by its own
// margin mk = vk inv_c inv_r (vk per segment, the exact path's formula): by
// its FP32 r when mk is within kTrust, else by a verification request (a
// full request buffer verifies it in place).  Adds go straight to the slab's
// shared-memory sums.  Returns the lane's number of requests.
__device__ __noinline__ int sum_near(Smem& sm, const float2 (&cov_end)[kDiags], int s, int t,
                                     bool fx, bool fy, float2 m, float2 vk) {
  const SlowCtx& cx = sm.cx;
  const int r0 = s * kRows;
  const int cb0 = 8 * (s + t);
  float2 c[kDiags];
#pragma unroll
  for (int k = 0; k < kDiags; ++k) c[k] = cov_end[k];
#pragma unroll 1
  for (int rr = kRows - 1; rr >= 0; --rr) {
    const float4 rf = sm.r_fg[r0 + rr];
#pragma unroll
    for (int k = 0; k < kDiags; ++k) {
      const float4 cf = col_fg(sm, padc(ringc(cx.ring0, cb0 + rr + k)));
      c[k] = fma2(make_float2(-rf.x, -rf.y), make_float2(cf.z, cf.w), c[k]);
      c[k] = fma2(make_float2(-cf.x, -cf.y), make_float2(rf.z, rf.w), c[k]);
    }
  }
  int nreq = 0;
  float tmax = 0.f;
#pragma unroll 1
  for (int rr = 0; rr < kRows; ++rr) {
    const float4 rf = sm.r_fg[r0 + rr];
    const float2 ivr = sm.r_iv[r0 + rr];
#pragma unroll 1
    for (int k = 0; k < kDiags; ++k) {
      const int rcx = ringc(cx.ring0, cb0 + rr + k);
      const int slot = padc(rcx);
      const float2 ivc = sm.u.s.c_iv[slot];
      const float2 r2 = mul2(mul2(c[k], ivc), ivr);
      const float2 mk2 = mul2(mul2(vk, ivc), ivr);
#pragma unroll 1
      for (int g = 0; g < 2; ++g) {
        const float r = g ? r2.y : r2.x;
        if (!((g ? fy : fx) && fabsf(r - cx.thr) <= (g ? m.y : m.x))) continue;  // NaN: skip
        const float mk = g ? mk2.y : mk2.x;
        float add = 0.f;
        if (mk <= kTrust) {
          if (r > cx.thr) {
            add = r;
            tmax = fmaxf(tmax, mk);
          }
        } else {
          const int64_t i = cx.rbase[g] + r0 + rr;
          const int64_t j = i + cx.D0 + t * kDiags + k;
          const unsigned long long sl = atomicAdd(cx.vcount, 1ull);
          ++nreq;
          if (sl < static_cast<unsigned long long>(cx.vcap)) {
            VerifyReq q;
            q.i = static_cast<uint64_t>(i) | (static_cast<uint64_t>(cx.prob) << 40);
            q.d = static_cast<uint32_t>(j - i);
            q.ub = r + mk;
            cx.vreq[sl] = q;
          } else {
            // request buffer full: verified in place (counted)
            const Problem& pr = *cx.pr;
            const float ev = (cov_part(pr.R, pr.C, i, j, 0, cx.m) * pr.C.inv32[j]) * pr.R.inv32[i];
            atomicAdd(cx.overflow, 1ull);
            if (ev > cx.thr) add = ev;
          }
        }
        if (add != 0.f) {
          atomicAdd(g ? &sm.r_best[r0 + rr].y : &sm.r_best[r0 + rr].x, add);
          atomicAdd(g ? &sm.c_best[padc(rcx)].y : &sm.c_best[padc(rcx)].x, add);
        }
      }
      const float4 cf = col_fg(sm, slot);
      c[k] = fma2(make_float2(cf.x, cf.y), make_float2(rf.z, rf.w), c[k]);
      c[k] = fma2(make_float2(rf.x, rf.y), make_float2(cf.z, cf.w), c[k]);
    }
  }
  if (tmax > 0.f) atomicMax(cx.tmargin, static_cast<unsigned long long>(__float_as_uint(tmax)));
  return nreq;
}

// Bounds pass: raises a row's or column's pair of bounds in shared memory
// (float bits of non-negative floats).
__device__ __forceinline__ void raise_shared(float2& slot, unsigned x, unsigned y) {
  const float2 old = slot;
  if (x > __float_as_uint(old.x)) atomicMax(reinterpret_cast<unsigned*>(&slot.x), x);
  if (y > __float_as_uint(old.y)) atomicMax(reinterpret_cast<unsigned*>(&slot.y), y);
}

// Raises window w's key to the bound lb > 0 (0: none; then w may lie outside
// the series).  The key carries no partner: its index field 0 loses every
// tie, and the cell the bound came from has a larger r, so a real cell
// replaces it.
// k-best lists (k > 0): every call's bound comes from cells of its own (a
// row's in one band, a column's in one unit), so a list of the largest k
// bounds holds a lower bound of the k-th best.
__device__ __forceinline__ void raise_bound(uint64_t* keys, int64_t w, float lb,
                                            const KeyLayout& kl, int k) {
  if (!keys || !(lb > 0.f)) return;
  const uint64_t key = q_from_float_bits(__float_as_uint(lb), kl.frac_bits) << kl.idx_bits;
  if (k > 0) {
    u64* list = reinterpret_cast<u64*>(keys + w * k);
    if (key > __ldcg(list + k - 1)) topk_insert(list, k, key);
  } else if (key > __ldcg(keys + w)) {
    atomicMax(reinterpret_cast<u64*>(keys + w), key);
  }
}

// MATRIX_SUMMARY: a thread's running maxima (per segment and target).
struct MatRun {
  int cell[2][2];
  float mx[2][2];
};

// MATRIX_SUMMARY: a thread-step whose block crosses a grid boundary (flags
// fx, fy per segment) is walked again from the step's start (rewound from
// the covariances at its end, as the exact path rewinds), and every cell
// above the threshold goes to its own grid entry.
__device__ __noinline__ void mat_cells_block(Smem& sm, const float2 (&cov_end)[kDiags], int s,
                                             int t, bool fx, bool fy) {
  const SlowCtx& cx = sm.cx;
  const int r0 = s * kRows;
  const int cb0 = 8 * (s + t);
  float2 c[kDiags];
#pragma unroll
  for (int k = 0; k < kDiags; ++k) c[k] = cov_end[k];
#pragma unroll 1
  for (int rr = kRows - 1; rr >= 0; --rr) {
    const float4 rf = sm.r_fg[r0 + rr];
#pragma unroll
    for (int k = 0; k < kDiags; ++k) {
      const float4 cf = col_fg(sm, padc(ringc(cx.ring0, cb0 + rr + k)));
      c[k] = fma2(make_float2(-rf.x, -rf.y), make_float2(cf.z, cf.w), c[k]);
      c[k] = fma2(make_float2(-cf.x, -cf.y), make_float2(rf.z, rf.w), c[k]);
    }
  }
#pragma unroll 1
  for (int rr = 0; rr < kRows; ++rr) {
    const float4 rf = sm.r_fg[r0 + rr];
    const float2 dfr = make_float2(rf.x, rf.y), dgr = make_float2(rf.z, rf.w);
    const float2 ivr = sm.r_iv[r0 + rr];
#pragma unroll
    for (int k = 0; k < kDiags; ++k) {
      const int slot = padc(ringc(cx.ring0, cb0 + rr + k));
      const float2 r2 = mul2(mul2(c[k], sm.u.s.c_iv[slot]), ivr);
#pragma unroll
      for (int g = 0; g < 2; ++g) {
        const float r = g ? r2.y : r2.x;
        if ((g ? fy : fx) && r > cx.thr) {  // false for NaN
          const int64_t i = cx.rbase[g] + r0 + rr;
          const int64_t j = i + cx.D0 + t * kDiags + k;
          if (cx.mcol)
            atomicMax(cx.mat + div_magic(i, cx.rpc_magic) * cx.mat_w + div_magic(j, cx.cpc_magic),
                      ord_float(r));
          if (cx.mrow)
            atomicMax(cx.mat + div_magic(j, cx.rpc_magic) * cx.mat_w + div_magic(i, cx.cpc_magic),
                      ord_float(r));
        }
      }
      const float4 cf = col_fg(sm, slot);
      c[k] = fma2(make_float2(cf.x, cf.y), dgr, c[k]);
      c[k] = fma2(dfr, make_float2(cf.z, cf.w), c[k]);
    }
  }
}

// The band kernel's body; kSum selects SUM_THRESH (separate instantiations,
// so the 1NN_INDEX form carries none of the sum bookkeeping).  kCoarse
// selects the fast path's filter:
//   false: per cell, r = (cov * inv_c) * inv_r, the block's largest r
//          against the threshold (8 packed multiplies per row);
//   true:  per step, the block's largest covariance times the largest
//          inverse norms of its columns and rows -- an upper bound of every
//          r in the block, which spares the per-cell multiplies.  It is
//          tight where the inverse norms of neighbouring windows are close
//          (long windows); a block it flags goes to the exact path, which
//          checks every cell with its own r.
// kMat selects MATRIX_SUMMARY (running grid maxima), kKnn the k-best lists
// (filters at each window's k-th best); both take the per-cell filter.
// kExact selects the FP64 1NN form: the FP32 arithmetic only rules cells out,
// by the deterministic bound E (kStepCov ...), and every other cell's r is
// computed in FP64 (verify_exact_kernel).
// kBound selects the bounds pass: every cell raises its row's and its
// column's best (kMat: its grid entry) to its FP32 r less the step's margin,
// a bound with no partner (no candidate is looked at, nothing is verified).
template <bool kSum, bool kCoarse, bool kMat = false, bool kKnn = false, bool kExact = false,
          bool kBound = false>
__device__ __forceinline__ void band_body(const JoinParams& P) {
  static_assert(!(kMat && (kSum || kCoarse)), "the matrix form takes per-cell maxima");
  static_assert(!(kKnn && (kSum || kCoarse || kMat)), "the k-best form is a 1NN variant");
  static_assert(!(kExact && (kSum || kKnn || kCoarse)), "no exact form of these");
  static_assert(!kBound || kExact, "bounds are the exact form's");
  constexpr bool kRaise = kBound && !kMat;   // bounds of every window
  constexpr bool kRuns = kMat && (!kExact || kBound);  // running maxima of grid entries
  constexpr bool kWindow = !kRaise && !(kSum && !kCoarse);  // steps carry the column window
  extern __shared__ __align__(16) unsigned char smem_raw[];
  Smem& sm = *reinterpret_cast<Smem*>(smem_raw);
  const int t = threadIdx.x;
  const int lane = t & 31, warp = t >> 5;
  constexpr bool sum_mode = kSum;
  const float thr = static_cast<float>(P.threshold);
  // a window's filter value: its best (1NN), or its list's k-th best, at
  // least the threshold (k-best lists of kk keys per window)
  const int kk = kKnn ? P.knn_k : 1;
  auto best_floor = [&](const uint64_t* keys, int64_t w) -> float {
    const float v = key_corr_floor(keys[w * kk + (kk - 1)], P.kl);
    return kKnn ? fmaxf(v, thr) : v;
  };
  unsigned long long n_steps = 0, n_slow = 0, n_verify = 0;
  int qn = 0;  // queued blocks of this warp (warp-uniform)
  float tfast = 0.f;  // SUM_THRESH: largest margin of a block added on the fast path
  // MATRIX_SUMMARY: per segment (x, y) and target (column, row results) the
  // grid entry the thread's recent blocks fell in and their largest r, kept
  // in the exact path's queue space (the matrix form queues nothing)
  static_assert(sizeof(MatRun) * kThreads <= sizeof(SlowItem) * kWarps * kQueue,
                "matrix state exceeds the queue space");
  MatRun& mrun = reinterpret_cast<MatRun*>(&sm.queue[0][0])[t];
  if constexpr (kRuns) {
#pragma unroll
    for (int g = 0; g < 2; ++g)
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        mrun.cell[g][h] = -1;
        mrun.mx[g][h] = -3.f;
      }
  }

  if (lane == 0) sm.rq_used[warp] = kReqChunk;  // no block of requests yet
  __syncwarp();
  // exact form: series out of FP32's safe range leave every unit to the FP64
  // band kernel
  bool out_of_range = false;
  if constexpr (kExact) {
    const float vmax = __uint_as_float(P.range[0]), imax = __uint_as_float(P.range[1]);
    out_of_range = !(vmax <= kExactMaxValue && imax <= kExactMaxInv && vmax * imax <= kExactMaxRatio);
  }

  for (;;) {
    if (t == 0) {
      const long long uu = static_cast<long long>(atomicAdd(P.unit_counter, 1ull));
      sm.unit = uu;
      if constexpr (kExact) {
        sm.cx.unit_reqs = 0;
        sm.cx.unit_wide = 0;
        sm.cx.unit_lost = 0;
        sm.cx.budget = P.req_budget;
        sm.cx.wide_budget = P.wide_budget;
        if (!kBound && out_of_range && uu < P.total_units)
          P.fp64_list[atomicAdd(P.fp64_count, 1ull)] = uu;  // (no request made)
      }
      if (uu < P.total_units) {
        int pi;
        int64_t bb, ubb;
        decode_unit(P, uu, &pi, &bb, &ubb);
        sm.prob = problem_of(P, pi);
        sm.prob_index = pi;
        sm.band = bb;
        sm.unit_in_band = ubb;
      }
    }
    __syncthreads();
    const int64_t u = sm.unit;
    if (u >= P.total_units) break;
    if constexpr (kExact) {
      if (out_of_range) {
        __syncthreads();  // sm.unit is read before the next fetch
        continue;
      }
    }
    if constexpr (kBound) {
      // (uniform: sm.prob, sm.band and sm.unit_in_band are the unit's)
      bool skip;
      if constexpr (kMat) {
        // rows of every grid entry: every second to eighth unit of a band
        const int64_t span = P.rows_per_cell < P.cols_per_cell ? P.rows_per_cell : P.cols_per_cell;
        int64_t stride = span / (2 * sm.prob.seg_len);
        stride = stride < 1 ? 1 : (stride > 8 ? 8 : stride);
        skip = sm.unit_in_band % stride != 0;
      } else {
        // about 2^14 cells per window; k-best lists: 4 k bands
        const int64_t longest = sm.prob.R.ns > sm.prob.C.ns ? sm.prob.R.ns : sm.prob.C.ns;
        int64_t stride = longest >> 14;
        if (P.knn_k && stride > longest / (int64_t{4} * kBand * P.knn_k))
          stride = longest / (int64_t{4} * kBand * P.knn_k);
        if (stride < 1) stride = 1;
        skip = sm.band % stride != stride - 1;
      }
      if (skip) {
        __syncthreads();
        continue;
      }
    }
    const Problem& pr = sm.prob;
    const int64_t K = pr.seg_len;  // per problem: batched joins mix windows
    const int64_t m = pr.m;
    const int64_t band = sm.band, ub = sm.unit_in_band;
    const int64_t D0 = pr.d_lo + band * kBand;
    const int64_t rows_b = band_rows(pr.R.ns, pr.C.ns, D0);
    int64_t seg_row[2], seg_len[2];
    seg_row[0] = ub * 2 * K;
    seg_row[1] = seg_row[0] + K;
#pragma unroll
    for (int g = 0; g < 2; ++g) {
      const int64_t l = rows_b - seg_row[g];
      seg_len[g] = l < 0 ? 0 : (l > K ? K : l);
    }
    const int64_t d_my = D0 + t * kDiags;
    const int sh = pr.C.bshift;

    // ---------------- anchors ----------------
    // With the thread's first column window j0 and
    // Y(p) = T32c[p] + (boff_c[p >> bshift] - mu_j0) (the column samples
    // centred by that window's mean, shared by the thread's 8 windows):
    //   anchor_k = sum_t xc_t * Y(j_k + t) - (mu_jk - mu_j0) * sum_t xc_t
    // where xc is the row window centred by its FP64 mean.  The two segments
    // run as f32x2 pairs: their column spans are seg_len apart, a multiple of
    // the block size, so both halves cross block boundaries together.  The
    // row windows and the CTA's column spans are staged in shared memory.
    float2 acc2[kDiags];
    float2 xsum2 = make_float2(0.f, 0.f);
    // exact form: squared norms of the row window and of the column samples,
    // and the thread's first window's FP64 mean per segment
    [[maybe_unused]] float2 x2 = make_float2(0.f, 0.f), y2 = make_float2(0.f, 0.f);
    [[maybe_unused]] double mu0d[2];
#pragma unroll
    for (int k = 0; k < kDiags; ++k) acc2[k] = make_float2(0.f, 0.f);
    int64_t jb[2], b0s[2];
    float mu0[2];
    float2 o0[2];                 // {bhi, blo} of the block of mu_j0
#pragma unroll
    for (int g = 0; g < 2; ++g) {
      jb[g] = seg_row[g] + d_my;  // the thread's first column window
      const int64_t jc = jb[g] < pr.C.ns ? jb[g] : pr.C.ns - 1;
      b0s[g] = jc >> sh;
      mu0[g] = pr.C.mu_rel[jc];   // mu_j0 - boff_c[b0]
      o0[g] = make_float2(pr.C.bhi[b0s[g]], pr.C.blo[b0s[g]]);
      if constexpr (kExact) mu0d[g] = pr.C.mean[jc];
    }
    const bool live1 = seg_len[1] > 0;
    const int64_t nblk_c = (pr.C.n + (int64_t{1} << sh) - 1) >> sh;
    int64_t span_b0 = 0;
    // anchors from the tensor-core table (anchor_tc.cu) when the join has one
    const bool tab = pr.anchor_tab != nullptr;
    if (tab) {
#pragma unroll
      for (int g = 0; g < 2; ++g) {
        const bool live = g == 0 ? seg_len[0] > 0 : live1;
        const float* rowp = pr.anchor_tab + (seg_row[g] / K - pr.tab_s0) * pr.tab_wp +
                            band * kBand + t;
#pragma unroll
        for (int k = 0; k < kDiags; ++k) {
          const float v = (live && jb[g] + k < pr.C.ns) ? rowp[k * 128] : 0.f;
          if (g) acc2[k].y = v; else acc2[k].x = v;
        }
      }
    }
    for (int64_t t0 = 0; t0 < (tab ? 0 : m); t0 += kAnchorChunk) {
      const int chunk = static_cast<int>((m - t0) < kAnchorChunk ? (m - t0) : kAnchorChunk);
      {
        const int64_t i0 = seg_row[0], i1 = seg_row[1];
        const int64_t bi0 = i0 >> sh, bi1 = i1 >> sh;
        const float mr0 = pr.R.mu_rel[i0], mr1 = live1 ? pr.R.mu_rel[i1] : 0.f;
        for (int x = t; x < chunk; x += kThreads) {
          const int64_t p0 = i0 + t0 + x, p1 = i1 + t0 + x;
          float2 v;
          if constexpr (kExact) {
            v.x = static_cast<float>(pr.R.T[p0] - pr.R.mean[i0]);
            v.y = live1 ? static_cast<float>(pr.R.T[p1] - pr.R.mean[i1]) : 0.f;
            sm.u.a.xr[x] = v;
            continue;
          }
          v.x = pr.R.T32[p0] + (block_delta(pr.R, p0 >> sh, bi0) - mr0);
          v.y = live1 ? pr.R.T32[p1] + (block_delta(pr.R, p1 >> sh, bi1) - mr1) : 0.f;
          sm.u.a.xr[x] = v;
        }
        const int64_t cb0 = i0 + D0 + t0, cb1 = i1 + D0 + t0;
        for (int x = t; x < kBand + chunk + 16; x += kThreads) {
          const int64_t p0 = cb0 + x, p1 = cb1 + x;
          float2 v;
          v.x = p0 < pr.C.n ? pr.C.T32[p0] : 0.f;
          v.y = (live1 && p1 < pr.C.n) ? pr.C.T32[p1] : 0.f;
          sm.u.a.yc[pady2(x)] = v;
        }
        if (t < 2 * kSpanBlk) {
          const int g = t >= kSpanBlk, x = t - g * kSpanBlk;
          const int64_t b = ((g ? cb1 : cb0) >> sh) + x;
          const bool ok = (g == 0 || live1) && b < nblk_c;
          if constexpr (kExact) sm.u.a.cbd[g][x] = ok ? pr.C.T[b << sh] : 0.0;
          else sm.u.a.cb[g][x] = ok ? make_float2(pr.C.bhi[b], pr.C.blo[b]) : make_float2(0.f, 0.f);
        }
        span_b0 = cb0 >> sh;
      }
      __syncthreads();
      const int64_t plim0 = pr.C.n;
      int64_t cur_b = -1;                        // block of the cached corrections
      float2 dlo = make_float2(0.f, 0.f), dhi = make_float2(0.f, 0.f);
      for (int c0 = 0; c0 < chunk; c0 += 32) {
        float2 part[kDiags];
#pragma unroll
        for (int k = 0; k < kDiags; ++k) part[k] = make_float2(0.f, 0.f);
        float2 xs = make_float2(0.f, 0.f);
        const int c1 = (c0 + 32 < chunk) ? c0 + 32 : chunk;
        // groups of 8 row samples: 16 column samples cover the 8 windows;
        // 16 consecutive samples touch at most two blocks (blocks hold >= 32)
        for (int xg = c0; xg < c1; xg += 8) {
          const int64_t pg = jb[0] + t0 + xg;
          const int64_t bf = pg >> sh;
          if (bf != cur_b) {
            // the same sums as block_delta(), from the staged offsets; the
            // second segment's blocks sit at the same span positions
            cur_b = bf;
            const int x = static_cast<int>(bf - span_b0);
            if constexpr (kExact) {
              // in FP64, rounded once
              dlo.x = (pg < plim0) ? static_cast<float>(sm.u.a.cbd[0][x] - mu0d[0]) : 0.f;
              dhi.x = (((bf + 1) << sh) < plim0)
                          ? static_cast<float>(sm.u.a.cbd[0][x + 1] - mu0d[0]) : 0.f;
              dlo.y = (live1 && pg + K < plim0) ? static_cast<float>(sm.u.a.cbd[1][x] - mu0d[1]) : 0.f;
              dhi.y = (live1 && ((bf + 1) << sh) + K < plim0)
                          ? static_cast<float>(sm.u.a.cbd[1][x + 1] - mu0d[1]) : 0.f;
            } else {
            const float2 l0 = sm.u.a.cb[0][x], h0 = sm.u.a.cb[0][x + 1];
            const float2 l1 = sm.u.a.cb[1][x], h1 = sm.u.a.cb[1][x + 1];
            dlo.x = (pg < plim0) ? ((l0.x - o0[0].x) + (l0.y - o0[0].y)) - mu0[0] : 0.f;
            dhi.x = (((bf + 1) << sh) < plim0) ? ((h0.x - o0[0].x) + (h0.y - o0[0].y)) - mu0[0] : 0.f;
            dlo.y = (live1 && pg + K < plim0) ? ((l1.x - o0[1].x) + (l1.y - o0[1].y)) - mu0[1] : 0.f;
            dhi.y = (live1 && ((bf + 1) << sh) + K < plim0)
                        ? ((h1.x - o0[1].x) + (h1.y - o0[1].y)) - mu0[1] : 0.f;
            }
          }
          const int nb = static_cast<int>(((bf + 1) << sh) - pg);  // samples left in block bf
          const int o = pady2(t * kDiags + xg);      // 16-byte aligned slot
          float2 y[16];
#pragma unroll
          for (int q = 0; q < 16; q += 2) {
            const float4 v = *reinterpret_cast<const float4*>(&sm.u.a.yc[o + q + (q >> 3) * 2]);
            y[q] = make_float2(v.x, v.y);
            y[q + 1] = make_float2(v.z, v.w);
          }
          if constexpr (kExact) {
            // the group's first 8 samples; all 16 in the window's last group
            const bool last = t0 + xg + 8 >= m;
#pragma unroll
            for (int q = 0; q < 8; ++q) y2 = fma2(y[q], y[q], y2);
            if (last) {
#pragma unroll
              for (int q = 8; q < 16; ++q) y2 = fma2(y[q], y[q], y2);
            }
            const float2 dm = make_float2(fmaxf(fabsf(dlo.x), fabsf(dhi.x)),
                                          fmaxf(fabsf(dlo.y), fabsf(dhi.y)));
            const float cnt = last ? 16.f : 8.f;
            y2 = fma2(mul2(make_float2(cnt, cnt), dm), dm, y2);
          }
#pragma unroll
          for (int q = 0; q < 16; ++q) {
            const float2 d = q < nb ? dlo : dhi;
            y[q] = make_float2(y[q].x + d.x, y[q].y + d.y);
          }
#pragma unroll
          for (int v = 0; v < 8; ++v) {
            if (xg + v < c1) {
              const float2 xv = sm.u.a.xr[xg + v];
              xs = make_float2(xs.x + xv.x, xs.y + xv.y);
              if constexpr (kExact) x2 = fma2(xv, xv, x2);
#pragma unroll
              for (int k = 0; k < kDiags; ++k) part[k] = fma2(xv, y[v + k], part[k]);
            }
          }
        }
#pragma unroll
        for (int k = 0; k < kDiags; ++k)
          acc2[k] = make_float2(acc2[k].x + part[k].x, acc2[k].y + part[k].y);
        xsum2 = make_float2(xsum2.x + xs.x, xsum2.y + xs.y);
      }
      __syncthreads();
    }
    [[maybe_unused]] float2 ekmax = make_float2(0.f, 0.f);
#pragma unroll
    for (int k = 0; k < kDiags; ++k) {
#pragma unroll
      for (int g = 0; g < 2; ++g) {
        const int64_t j = jb[g] + k;
        if (tab || j >= pr.C.ns || (g == 1 && !live1)) continue;
        if constexpr (kExact) {
          const float e = static_cast<float>(pr.C.mean[j] - mu0d[g]);
          if (g) {
            acc2[k].y = fmaf(-e, xsum2.y, acc2[k].y);
            ekmax.y = fmaxf(ekmax.y, fabsf(e));
          } else {
            acc2[k].x = fmaf(-e, xsum2.x, acc2[k].x);
            ekmax.x = fmaxf(ekmax.x, fabsf(e));
          }
          continue;
        }
        const float ek = (pr.C.mu_rel[j] + block_delta(pr.C, j >> sh, b0s[g])) - mu0[g];
        if (g) acc2[k].y = fmaf(-ek, xsum2.y, acc2[k].y);
        else acc2[k].x = fmaf(-ek, xsum2.x, acc2[k].x);
      }
    }
    float2 cov[kDiags];
#pragma unroll
    for (int k = 0; k < kDiags; ++k) {
      const int64_t d = d_my + k;
      const bool valid = d < pr.d_hi && !(d >= pr.x_lo && d < pr.x_hi);
      // An excluded diagonal carries NaN: every r on it is NaN and never wins.
      cov[k] = valid ? acc2[k] : make_float2(qnan(), qnan());
    }
    // Drift state of the thread, per segment: the sum over steps of the
    // largest cov^2 among its diagonals (an upper bound of every diagonal's
    // own sum), starting from the anchors' rounding; and the sum of squared
    // increment bounds.
    float2 Vt;  // (the exact form's bound E)
    if constexpr (kExact) {
      const float fm = static_cast<float>(m);
      Vt = make_float2(anchor_bound(x2.x, y2.x, ekmax.x, fm), anchor_bound(x2.y, y2.y, ekmax.y, fm));
    } else {
      const float2 cm = absmax8(cov);
      Vt = make_float2(pr.anchor_vcoef * cm.x * cm.x, pr.anchor_vcoef * cm.y * cm.y);
    }
    float2 W = make_float2(0.f, 0.f);

    if (t == 0) {
      // read by the exact path only after the slab's first barrier
      SlowCtx& cx = sm.cx;
      cx.pr = &sm.prob;
      cx.key_row = pr.key_row;
      cx.key_col = pr.key_col;
      cx.D0 = D0;
      cx.m = m;
      cx.kl = P.kl;
      cx.prob = sm.prob_index;
      cx.vreq = P.vreq;
      cx.vcount = P.counters + 3;
      cx.vcap = P.vreq_cap;
      cx.tmargin = P.counters + 4;
      cx.overflow = P.counters + 6;
      cx.sum_mode = kSum;
      cx.thr = static_cast<float>(P.threshold);
      cx.knn_k = kKnn || kExact ? P.knn_k : 0;
      if constexpr (kMat) {
        cx.mat = P.mat;
        cx.mat_w = P.mat_w;
        cx.mat_h = P.mat_h;
        cx.rpc = P.rows_per_cell;
        cx.cpc = P.cols_per_cell;
        cx.rpc_magic = P.rpc_magic;
        cx.cpc_magic = P.cpc_magic;
        cx.mcol = P.mat_col[sm.prob_index] != 0;
        cx.mrow = P.mat_row[sm.prob_index] != 0;
      }
    }

    // ---------------- slabs ----------------
    const int64_t nslabs = (seg_len[0] + kSlab - 1) / kSlab;
    for (int64_t q = 0; q < nslabs; ++q) {
      // steps with rows of the segment (whole pairs), and the staged columns
      // that they reach (sums and bounds: later slabs stage every entering
      // column, which flushes the previous one in its place)
      const int64_t left = seg_len[0] - q * kSlab;
      const int nsteps = left >= kSlab ? kSteps : static_cast<int>((left + 15) / 16) * 2;
      const int ncols = (kSum || kRaise) && q > 0 ? kCols : (kBand + nsteps * kRows + 31) / 32 * 32;
      int64_t rbase[2], rend[2], cbase_g[2];
#pragma unroll
      for (int g = 0; g < 2; ++g) {
        rbase[g] = seg_row[g] + q * kSlab;
        rend[g] = seg_row[g] + seg_len[g];
        cbase_g[g] = rbase[g] + D0;
        if (t == 0) sm.cx.rbase[g] = rbase[g];
      }
      const int ring0 = static_cast<int>((q * kSlab) % kCols);
      const int rq = ring0 >> 3;  // ring block of the slab's first column
      if (t == 0) sm.cx.ring0 = ring0;
      // Staging, coalesced: thread t stages columns t, t + kThreads, ... and
      // row t.  The filter tables are reduced on the way, 8 lanes (8
      // consecutive columns or rows) at a time: per 8-column block and per
      // 8-row step the smallest best, the largest inverse norm and the
      // largest |df|, |dg|.
      if (!sum_mode && !kRaise && q > 0 && P.refresh_cols && pr.key_col) {
        // Joins that start cold (no seeds): the columns kept from the last
        // slab take their bests from the profile keys, which other CTAs
        // raise quickly at the start; ring columns otherwise keep the bests
        // staged when they entered.
#pragma unroll 2
        for (int c = t; c < kCols - kSlab; c += kThreads) {
          const int rc = ringc(ring0, c);
          float2 cb = sm.c_best[padc(rc)];
          if (cb.x != kNoTarget) cb.x = fmaxf(cb.x, best_floor(pr.key_col, cbase_g[0] + c));
          if (cb.y != kNoTarget) cb.y = fmaxf(cb.y, best_floor(pr.key_col, cbase_g[1] + c));
          sm.c_best[padc(rc)] = cb;
          float2 mn = cb;
#pragma unroll
          for (int o = 1; o < 8; o <<= 1) {
            mn.x = fminf(mn.x, __shfl_xor_sync(0xffffffffu, mn.x, o));
            mn.y = fminf(mn.y, __shfl_xor_sync(0xffffffffu, mn.y, o));
          }
          if ((lane & 7) == 0) {
            const int b = rc >> 3;
            sm.c_blkmin[b] = mn;
            if (b == 0) sm.c_blkmin[kBlocks] = mn;
          }
        }
      }
#pragma unroll 3
      for (int c = (q == 0 ? 0 : kCols - kSlab) + t; c < ncols; c += kThreads) {
        const int rc = ringc(ring0, c);
        const int64_t j0 = cbase_g[0] + c, j1 = cbase_g[1] + c;
        const bool ok0 = seg_len[0] > 0 && j0 < pr.C.ns;
        const bool ok1 = seg_len[1] > 0 && j1 < pr.C.ns;
        float4 f;
        f.x = ok0 ? pr.C.df32[j0] : 0.f;
        f.y = ok1 ? pr.C.df32[j1] : 0.f;
        f.z = ok0 ? pr.C.dg32[j0] : 0.f;
        f.w = ok1 ? pr.C.dg32[j1] : 0.f;
        const float2 iv = make_float2(ok0 ? pr.C.inv32[j0] : qnan(), ok1 ? pr.C.inv32[j1] : qnan());
        // A window that cannot match (padding, NaN or flat) must not lower
        // the filter threshold: its best is "unreachable".
        float2 cbv;
        if constexpr (kRaise) {
          // the previous occupant's bounds go to its keys
          if (q > 0) {
            const float2 old = sm.c_best[padc(rc)];
            raise_bound(pr.key_col, j0 - kCols, old.x, P.kl, P.knn_k);
            raise_bound(pr.key_col, j1 - kCols, old.y, P.kl, P.knn_k);
          }
          cbv = make_float2(0.f, 0.f);
        } else if (sum_mode) {
          // the ring column's previous occupant (kCols columns earlier)
          // leaves: its sums go to the profile, the new one starts at 0
          if (q > 0 && pr.sum_col) {
            const float2 old = sm.c_best[padc(rc)];
            const int64_t o0 = j0 - kCols, o1 = j1 - kCols;
            if (old.x != 0.f && o0 >= 0 && o0 < pr.C.ns) atomicAdd(pr.sum_col + o0, static_cast<double>(old.x));
            if (old.y != 0.f && o1 >= 0 && o1 < pr.C.ns) atomicAdd(pr.sum_col + o1, static_cast<double>(old.y));
          }
          cbv = make_float2(0.f, 0.f);
        } else {
          cbv.x = (pr.key_col && ok0 && !isnan(iv.x)) ? best_floor(pr.key_col, j0) : kNoTarget;
          cbv.y = (pr.key_col && ok1 && !isnan(iv.y)) ? best_floor(pr.key_col, j1) : kNoTarget;
        }
        sm.u.s.c_df[padc(rc)] = make_float2(f.x, f.y);
        sm.u.s.c_dg[padc(rc)] = make_float2(f.z, f.w);
        sm.u.s.c_iv[padc(rc)] = iv;
        if (rc < kGhost) {
          sm.u.s.c_df[padc(rc + kCols)] = make_float2(f.x, f.y);
          sm.u.s.c_dg[padc(rc + kCols)] = make_float2(f.z, f.w);
          sm.u.s.c_iv[padc(rc + kCols)] = iv;
        }
        sm.c_best[padc(rc)] = cbv;
        TableEntry e = table_entry(f, iv, cbv);
        if constexpr (kExact) floor_dg(e);
        reduce8(e);  // 8 lanes = one aligned ring block
        if ((lane & 7) == 0) {
          const int b = rc >> 3;
          sm.c_blkmin[b] = e.mn;
          sm.c_blkmax_iv[b] = e.mx;
          sm.c_blkmax_fg[b] = e.mf;
          if (b == 0) {
            sm.c_blkmin[kBlocks] = e.mn;
            sm.c_blkmax_iv[kBlocks] = e.mx;
            sm.c_blkmax_fg[kBlocks] = e.mf;
          }
        }
      }
      {
        const int r = t;  // kSlab == kThreads
        const int64_t i0 = rbase[0] + r, i1 = rbase[1] + r;
        const bool ok0 = i0 < rend[0], ok1 = i1 < rend[1];
        float4 f;
        f.x = ok0 ? pr.R.df32[i0] : 0.f;
        f.y = ok1 ? pr.R.df32[i1] : 0.f;
        f.z = ok0 ? pr.R.dg32[i0] : 0.f;
        f.w = ok1 ? pr.R.dg32[i1] : 0.f;
        const float2 iv = make_float2(ok0 ? pr.R.inv32[i0] : qnan(), ok1 ? pr.R.inv32[i1] : qnan());
        float2 rbv;
        if (sum_mode || kRaise) {
          rbv = make_float2(0.f, 0.f);
        } else {
          rbv.x = (pr.key_row && ok0 && !isnan(iv.x)) ? best_floor(pr.key_row, i0) : kNoTarget;
          rbv.y = (pr.key_row && ok1 && !isnan(iv.y)) ? best_floor(pr.key_row, i1) : kNoTarget;
        }
        sm.r_fg[r] = f;
        sm.r_iv[r] = iv;
        sm.r_best[r] = rbv;
        TableEntry e = table_entry(f, iv, rbv);
        if constexpr (kExact) floor_dg(e);
        reduce8(e);
        if ((lane & 7) == 0) {
          sm.r_stepmin[r >> 3] = e.mn;
          sm.r_stepmax_iv[r >> 3] = e.mx;
          sm.r_stepmax_fg[r >> 3] = e.mf;
        }
      }
      __syncthreads();
      // ---------------- steps ----------------
      // Steps run in pairs.  The thread's column window is carried from the
      // first step of a pair to the second (the last 7 columns of step s are
      // the first 7 of step s + 1): column x of step s sits in slot
      // (8 * (s & 1) + x) & 15, so every slot index is a constant.  The exact
      // path runs only between pairs: a step whose trigger finds the warp's
      // queue full is recorded in `pend` and queued after the pair as a
      // two-step (or one-step) block.
      float4 cfw[16];
      float2 ciw[16];
      // bounds pass: the last 7 columns' bounds of a step, its next step's first
      [[maybe_unused]] float2 cnext[kDiags - 1];
      if constexpr (kRaise) {
#pragma unroll
        for (int x = 0; x < kDiags - 1; ++x) cnext[x] = make_float2(0.f, 0.f);
      }
      int pend = -1;
      // segments of the pending block, per step (bits 0-1, 2-3; SUM_THRESH,
      // every segment otherwise)
      int pmsk = 15;
      float2 vlast = make_float2(0.f, 0.f);
      auto step = [&](const int s, auto parity) {
        [[maybe_unused]] constexpr int P = decltype(parity)::value;
        const int r0 = s * kRows;
        // ring block of the step's first column 8(s + t)
        const int rb = (rq + s + t) < kBlocks ? (rq + s + t) : (rq + s + t - kBlocks);
        const int base = 9 * rb;  // its padded slot
        // filter threshold and margin: the step's 15 columns lie in ring
        // blocks rb and rb + 1
        const float2 bm0 = sm.c_blkmin[rb], bm1 = sm.c_blkmin[rb + 1];
        const float2 bm = make_float2(fminf(bm0.x, bm1.x), fminf(bm0.y, bm1.y));
        const float2 rsm = sm.r_stepmin[s];
        const float2 ic0 = sm.c_blkmax_iv[rb], ic1 = sm.c_blkmax_iv[rb + 1];
        const float2 icm = make_float2(fmaxf(ic0.x, ic1.x), fmaxf(ic0.y, ic1.y));
        const float2 irm = sm.r_stepmax_iv[s];
        [[maybe_unused]] float2 dE = make_float2(0.f, 0.f);  // exact form: the step's share of E
        {
          const float2 cm = absmax8(cov);
          if constexpr (kExact) dE = mul2(make_float2(kStepCov, kStepCov), cm);
          else Vt = fma2(cm, cm, Vt);
        }
        {
          // bound of |df_c dg_r| + |df_r dg_c| over the step's cells
          const float4 cf0 = sm.c_blkmax_fg[rb], cf1 = sm.c_blkmax_fg[rb + 1];
          const float4 cfm = make_float4(fmaxf(cf0.x, cf1.x), fmaxf(cf0.y, cf1.y),
                                         fmaxf(cf0.z, cf1.z), fmaxf(cf0.w, cf1.w));
          const float4 rfm = sm.r_stepmax_fg[s];
          const float2 inc = fma2(make_float2(rfm.x, rfm.y), make_float2(cfm.z, cfm.w),
                                  mul2(make_float2(rfm.z, rfm.w), make_float2(cfm.x, cfm.y)));
          if constexpr (kExact) {
            dE = fma2(make_float2(kStepInc, kStepInc), inc, dE);
            Vt = make_float2(Vt.x + dE.x, Vt.y + dE.y);
          } else {
            W = fma2(inc, inc, W);
          }
        }
        // (exact form: E with the roundings of the exact path's steps back)
        const float vx = kExact ? Vt.x + dE.x : Vt.x + W.x;
        const float vy = kExact ? Vt.y + dE.y : Vt.y + W.y;
        // threshold - margin, the margin as the exact path forms it per cell
        // (C eps sqrt(rows v) inv_c inv_r) but with the block's largest
        // inverse norms, an approximate square root and a 2^-16 allowance
        // for both
        const float2 mg = kExact ? mul2(mul2(Vt, icm), irm)
                                 : mul2(mul2(make_float2(sqrt_approx(vx), sqrt_approx(vy)), icm), irm);
        const float2 tb = sum_mode ? make_float2(thr, thr)
                                   : make_float2(fminf(bm.x, rsm.x), fminf(bm.y, rsm.y));
        constexpr float kMg = kExact ? kBoundSlack : kStepMarginC;
        const float2 tt = fma2(make_float2(-kMg, -kMg), mg, tb);
        const float tx = kExact ? tt.x - kAbsSlack : tt.x, ty = kExact ? tt.y - kAbsSlack : tt.y;

        // fast path: recurrence + block maximum
        float bx = -3.f, by = -3.f;
        if constexpr (kRaise) {
          // largest r of each row (over the thread's diagonals) and column
          float2 cmax[kRows + kDiags - 1];
          float4 cf[kRows + kDiags - 1];
          float2 ci[kRows + kDiags - 1];
          unsigned rmx = 0, rmy = 0;  // lane rr: row rr's bound over the warp (float bits)
          const float2 lo = make_float2(fmaf(kBoundSlack, mg.x, kAbsSlack),
                                        fmaf(kBoundSlack, mg.y, kAbsSlack));
#pragma unroll
          for (int x = 0; x < kRows + kDiags - 1; ++x) cmax[x] = make_float2(-3.f, -3.f);
#pragma unroll
          for (int x = 0; x < kDiags - 1; ++x) {
            cf[x] = col_fg(sm, base + x);
            ci[x] = sm.u.s.c_iv[base + x];
          }
#pragma unroll
          for (int rr = 0; rr < kRows; ++rr) {
            {
              const int x = rr + kDiags - 1;
              cf[x] = col_fg(sm, base + x + (x >> 3));
              ci[x] = sm.u.s.c_iv[base + x + (x >> 3)];
            }
            const float4 rf = sm.r_fg[r0 + rr];
            const float2 dfr = make_float2(rf.x, rf.y), dgr = make_float2(rf.z, rf.w);
            const float2 ivr = sm.r_iv[r0 + rr];
            float mx = -3.f, my = -3.f;
#pragma unroll
            for (int k = 0; k < kDiags; k += 2) {
              const int x = rr + k;
              const float2 ra = mul2(mul2(cov[k], ci[x]), ivr);
              const float2 rc = mul2(mul2(cov[k + 1], ci[x + 1]), ivr);
              mx = max3(mx, ra.x, rc.x);
              my = max3(my, ra.y, rc.y);
              cmax[x] = make_float2(fmaxf(cmax[x].x, ra.x), fmaxf(cmax[x].y, ra.y));
              cmax[x + 1] = make_float2(fmaxf(cmax[x + 1].x, rc.x), fmaxf(cmax[x + 1].y, rc.y));
            }
            // non-negative floats order as their bits (NaN gives 0)
            const unsigned ux = __reduce_max_sync(0xffffffffu, __float_as_uint(fmaxf(mx - lo.x, 0.f)));
            const unsigned uy = __reduce_max_sync(0xffffffffu, __float_as_uint(fmaxf(my - lo.y, 0.f)));
            if (lane == rr) {
              rmx = ux;
              rmy = uy;
            }
#pragma unroll
            for (int k = 0; k < kDiags; ++k) {
              const float4 c4 = cf[rr + k];
              cov[k] = fma2(make_float2(c4.x, c4.y), dgr, cov[k]);
              cov[k] = fma2(dfr, make_float2(c4.z, c4.w), cov[k]);
            }
          }
          if (lane < kRows) raise_shared(sm.r_best[r0 + lane], rmx, rmy);
#pragma unroll
          for (int x = 0; x < kRows + kDiags - 1; ++x)
            cmax[x] = make_float2(fmaxf(cmax[x].x - lo.x, 0.f), fmaxf(cmax[x].y - lo.y, 0.f));
#pragma unroll
          for (int x = 0; x < kDiags; ++x) {
            float2 v = cmax[x];
            if (x < kDiags - 1) v = make_float2(fmaxf(v.x, cnext[x].x), fmaxf(v.y, cnext[x].y));
            raise_shared(sm.c_best[base + x], __float_as_uint(v.x), __float_as_uint(v.y));
          }
#pragma unroll
          for (int x = 0; x < kDiags - 1; ++x) cnext[x] = cmax[kDiags + x];
        } else if constexpr (kCoarse) {
          // largest covariance of the block (NaN diagonals ignored), then
          // the bound max(cov, 0) * max inv_c * max inv_r of every r in it
#pragma unroll
          for (int rr = 0; rr < kRows; ++rr) {
            {
              const int x = rr + kDiags - 1;
              cfw[(8 * P + x) & 15] = col_fg(sm, base + x + (x >> 3));
            }
            const float4 rf = sm.r_fg[r0 + rr];
            const float2 dfr = make_float2(rf.x, rf.y), dgr = make_float2(rf.z, rf.w);
            {
              const float ax = max3(cov[0].x, cov[1].x, cov[2].x);
              const float ay = max3(cov[0].y, cov[1].y, cov[2].y);
              const float cx3 = max3(cov[3].x, cov[4].x, cov[5].x);
              const float cy3 = max3(cov[3].y, cov[4].y, cov[5].y);
              bx = max3(bx, cov[6].x, cov[7].x);
              by = max3(by, cov[6].y, cov[7].y);
              bx = max3(bx, ax, cx3);
              by = max3(by, ay, cy3);
            }
#pragma unroll
            for (int k = 0; k < kDiags; ++k) {
              const float4 c4 = cfw[(8 * P + rr + k) & 15];
              cov[k] = fma2(make_float2(c4.x, c4.y), dgr, cov[k]);
              cov[k] = fma2(dfr, make_float2(c4.z, c4.w), cov[k]);
            }
          }
          const float2 bnd = mul2(mul2(make_float2(fmaxf(bx, 0.f), fmaxf(by, 0.f)), icm), irm);
          bx = bnd.x;
          by = bnd.y;
        } else if constexpr (kSum) {
          // SUM_THRESH: every cell's r (rounded as the exact path rounds it)
          // against the threshold, where the segment's step margin is within
          // kTrust (elsewhere `the` is out of reach and the segment goes to
          // the exact path if it reaches the threshold); row sums per step
          // row, column sums per step column, reduced after the step.  The
          // column values come straight from shared memory (no carried
          // window: its registers hold the sums).
          // a cell above the threshold by more than the step's margin (which
          // bounds every cell's own margin) adds its r; cells within it are
          // rare and settled by sum_near after the step
          const float2 smg = mul2(make_float2(kStepMarginC, kStepMarginC), mg);
          const float thx = thr + smg.x, thy = thr + smg.y;
          float2 dmin = make_float2(3.f, 3.f);  // nearest |r - thr| of the step
          float2 rsum[kRows];
          float2 cacc[kRows + kDiags - 1];
#pragma unroll
          for (int x = 0; x < kRows + kDiags - 1; ++x) cacc[x] = make_float2(0.f, 0.f);
#pragma unroll
          for (int rr = 0; rr < kRows; ++rr) {
            const float4 rf = sm.r_fg[r0 + rr];
            const float2 dfr = make_float2(rf.x, rf.y), dgr = make_float2(rf.z, rf.w);
            const float2 ivr = sm.r_iv[r0 + rr];
            rsum[rr] = make_float2(0.f, 0.f);
            float2 rodd;  // the previous diagonal's r (k odd)
#pragma unroll
            for (int k = 0; k < kDiags; ++k) {
              const int x = rr + k;
              const int slot = base + x + (x >> 3);
              const float4 c4 = col_fg(sm, slot);
              const float2 r2 = mul2(mul2(cov[k], sm.u.s.c_iv[slot]), ivr);
              // (two cells per three-input instruction; NaN cells are ignored)
              if (k & 1) {
                bx = max3(bx, rodd.x, r2.x);
                by = max3(by, rodd.y, r2.y);
                dmin = make_float2(min3(dmin.x, fabsf(rodd.x - thr), fabsf(r2.x - thr)),
                                   min3(dmin.y, fabsf(rodd.y - thr), fabsf(r2.y - thr)));
              } else {
                rodd = r2;
              }
              const float ax = r2.x > thx ? r2.x : 0.f;
              const float ay = r2.y > thy ? r2.y : 0.f;
              rsum[rr] = make_float2(rsum[rr].x + ax, rsum[rr].y + ay);
              cacc[x] = make_float2(cacc[x].x + ax, cacc[x].y + ay);
              cov[k] = fma2(make_float2(c4.x, c4.y), dgr, cov[k]);
              cov[k] = fma2(dfr, make_float2(c4.z, c4.w), cov[k]);
            }
          }
          // rows: a reduce-scatter over the warp (lanes 4 r .. 4 r + 3 end
          // with row r's total), one shared-memory atomic per row
          {
            float2 w4[4], w2[2];
            const bool b16 = lane & 16, b8 = lane & 8, b4 = lane & 4;
#pragma unroll
            for (int i = 0; i < 4; ++i) {
              const float2 snd = b16 ? rsum[i] : rsum[i + 4];
              const float2 kp = b16 ? rsum[i + 4] : rsum[i];
              w4[i] = make_float2(kp.x + __shfl_xor_sync(0xffffffffu, snd.x, 16),
                                  kp.y + __shfl_xor_sync(0xffffffffu, snd.y, 16));
            }
#pragma unroll
            for (int i = 0; i < 2; ++i) {
              const float2 snd = b8 ? w4[i] : w4[i + 2];
              const float2 kp = b8 ? w4[i + 2] : w4[i];
              w2[i] = make_float2(kp.x + __shfl_xor_sync(0xffffffffu, snd.x, 8),
                                  kp.y + __shfl_xor_sync(0xffffffffu, snd.y, 8));
            }
            const float2 snd = b4 ? w2[0] : w2[1];
            float2 z = b4 ? w2[1] : w2[0];
            z.x += __shfl_xor_sync(0xffffffffu, snd.x, 4);
            z.y += __shfl_xor_sync(0xffffffffu, snd.y, 4);
            z.x += __shfl_xor_sync(0xffffffffu, z.x, 2);
            z.y += __shfl_xor_sync(0xffffffffu, z.y, 2);
            z.x += __shfl_xor_sync(0xffffffffu, z.x, 1);
            z.y += __shfl_xor_sync(0xffffffffu, z.y, 1);
            const int row = (b16 ? 4 : 0) + (b8 ? 2 : 0) + (b4 ? 1 : 0);
            if ((lane & 3) == 0) {
              if (z.x != 0.f) atomicAdd(&sm.r_best[r0 + row].x, z.x);
              if (z.y != 0.f) atomicAdd(&sm.r_best[r0 + row].y, z.y);
            }
          }
          // columns: thread t's step columns 8..14 are thread t + 1's 0..6
#pragma unroll
          for (int x = 0; x < kDiags - 1; ++x) {
            const float ux = __shfl_up_sync(0xffffffffu, cacc[8 + x].x, 1);
            const float uy = __shfl_up_sync(0xffffffffu, cacc[8 + x].y, 1);
            if (lane > 0) cacc[x] = make_float2(cacc[x].x + ux, cacc[x].y + uy);
          }
          // (padded slots: at a stride of 9 pairs the lanes meet no bank conflict)
#pragma unroll
          for (int x = 0; x < kRows; ++x) {
            float2& cs = sm.c_best[base + x];
            if (cacc[x].x != 0.f) atomicAdd(&cs.x, cacc[x].x);
            if (cacc[x].y != 0.f) atomicAdd(&cs.y, cacc[x].y);
          }
          if (lane == 31) {
            const int next = rb + 1 < kBlocks ? base + 9 : 0;
#pragma unroll
            for (int x = 0; x < kDiags - 1; ++x) {
              float2& cs = sm.c_best[next + x];
              if (cacc[8 + x].x != 0.f) atomicAdd(&cs.x, cacc[8 + x].x);
              if (cacc[8 + x].y != 0.f) atomicAdd(&cs.y, cacc[8 + x].y);
            }
          }
          const bool nx = dmin.x <= smg.x, ny = dmin.y <= smg.y;
          if (nx || ny) {
            const float2 vk = make_float2(kBoundC * kEps * sqrtf(kRows * vx),
                                          kBoundC * kEps * sqrtf(kRows * vy));
            n_verify += sum_near(sm, cov, s, t, nx, ny, smg, vk);
          }
          // the largest margin of a value added from FP32 by this step
          if (bx > thx) tfast = fmaxf(tfast, smg.x);
          if (by > thy) tfast = fmaxf(tfast, smg.y);
        } else {
          float2 rprev;
#pragma unroll
          for (int rr = 0; rr < kRows; ++rr) {
            {
              const int x = rr + kDiags - 1;
              cfw[(8 * P + x) & 15] = col_fg(sm, base + x + (x >> 3));
              ciw[(8 * P + x) & 15] = sm.u.s.c_iv[base + x + (x >> 3)];
            }
            const float4 rf = sm.r_fg[r0 + rr];
            const float2 dfr = make_float2(rf.x, rf.y), dgr = make_float2(rf.z, rf.w);
            const float2 ivr = sm.r_iv[r0 + rr];
            // the row's largest cov * inv_c, times inv_r (> 0): the largest r
            // of the row, rounded exactly as (cov * inv_c) * inv_r per cell.
            // (From -3 the result is an upper bound only: -3 inv_r where every
            // r of the row lies below that.  A filter may take it; a grid
            // entry's maximum and its lower bound have to be a cell's r, and
            // a row without a cell leaves bx, by at -3.)
            float mx = kMat ? -INFINITY : -3.f, my = mx;
#pragma unroll
            for (int k = 0; k < kDiags; k += 2) {
              const float2 pa = mul2(cov[k], ciw[(8 * P + rr + k) & 15]);
              const float2 pb = mul2(cov[k + 1], ciw[(8 * P + rr + k + 1) & 15]);
              mx = max3(mx, pa.x, pb.x);
              my = max3(my, pa.y, pb.y);
            }
            const float2 rm = mul2(make_float2(mx, my), ivr);
            if (rr & 1) {
              bx = max3(bx, rprev.x, rm.x);
              by = max3(by, rprev.y, rm.y);
            } else {
              rprev = rm;
            }
#pragma unroll
            for (int k = 0; k < kDiags; ++k) {
              const float4 c4 = cfw[(8 * P + rr + k) & 15];
              cov[k] = fma2(make_float2(c4.x, c4.y), dgr, cov[k]);
              cov[k] = fma2(dfr, make_float2(c4.z, c4.w), cov[k]);
            }
          }
        }
        [[maybe_unused]] bool trig = bx > tx || by > ty;
        if constexpr (kMat && kExact && !kBound) {
          // exact matrix: a block that may hold a grid entry's largest r, by
          // the bounds of the entries it touches (two each way at most)
          trig = false;
#pragma unroll
          for (int g = 0; g < 2; ++g) {
            const float ub = (g ? by : bx) + fmaf(kBoundSlack, g ? mg.y : mg.x, kAbsSlack);
            if (!(ub > thr)) continue;
            const int64_t i0 = rbase[g] + r0, j0 = i0 + d_my;
            if (i0 >= pr.R.ns || j0 >= pr.C.ns) continue;  // no cell, no grid entry
            float lo = kNoTarget;
            if (sm.cx.mcol) lo = mat_block_floor(sm.cx, i0, kRows - 1, j0, kRows + kDiags - 2);
            if (sm.cx.mrow)
              lo = fminf(lo, mat_block_floor(sm.cx, j0, kRows + kDiags - 2, i0, kRows - 1));
            trig = trig || ub > lo;
          }
        } else if constexpr (kMat) {
          // a block inside one grid entry (per target) raises the thread's
          // running maximum of that entry, published when the thread's
          // blocks move on; a block across a grid boundary routes each cell
          trig = false;
          const float2 smg = mul2(make_float2(kMg, kMg), mg);
          // the exact form's bounds lie E below the values
          const float2 sub = kExact ? make_float2(smg.x + kAbsSlack, smg.y + kAbsSlack)
                                    : make_float2(0.f, 0.f);
          bool nonuni[2] = {false, false};
#pragma unroll
          for (int g = 0; g < 2; ++g) {
            const float bm = (g ? by : bx) - (g ? sub.y : sub.x);
            if (!((g ? by : bx) > -3.f && bm > thr)) continue;
            const int64_t i0 = rbase[g] + r0, j0 = i0 + d_my;
            if (i0 >= pr.R.ns || j0 >= pr.C.ns) continue;  // no cell, no grid entry
            tfast = fmaxf(tfast, g ? smg.y : smg.x);
            const int64_t rpc = sm.cx.rpc, cpc = sm.cx.cpc;
            int cell[2] = {-1, -1};
            bool uni = true;
            if (sm.cx.mcol) {
              const int64_t qa = div_magic(i0, sm.cx.rpc_magic), qb = div_magic(j0, sm.cx.cpc_magic);
              uni = uni && i0 - qa * rpc + (kRows - 1) < rpc &&
                    j0 - qb * cpc + (kRows + kDiags - 2) < cpc;
              cell[0] = static_cast<int>(qa * sm.cx.mat_w + qb);
            }
            if (sm.cx.mrow) {
              const int64_t qa = div_magic(j0, sm.cx.rpc_magic), qb = div_magic(i0, sm.cx.cpc_magic);
              uni = uni && j0 - qa * rpc + (kRows + kDiags - 2) < rpc &&
                    i0 - qb * cpc + (kRows - 1) < cpc;
              cell[1] = static_cast<int>(qa * sm.cx.mat_w + qb);
            }
            if (!uni) {
              nonuni[g] = true;
              continue;
            }
#pragma unroll
            for (int h = 0; h < 2; ++h) {
              if (cell[h] < 0) continue;
              const int cur = mrun.cell[g][h];
              if (cell[h] != cur) {
                if (cur >= 0) atomicMax(sm.cx.mat + cur, ord_float(mrun.mx[g][h]));
                mrun.cell[g][h] = cell[h];
                mrun.mx[g][h] = bm;
              } else {
                mrun.mx[g][h] = fmaxf(mrun.mx[g][h], bm);
              }
            }
          }
          // (the bounds pass does without the blocks across a boundary: their
          // cells one by one took two thirds of its time)
          if (!kBound && (nonuni[0] || nonuni[1]))
            mat_cells_block(sm, cov, s, t, nonuni[0], nonuni[1]);
        }
        // segments the exact path walks (bit 0: first, bit 1: second)
        [[maybe_unused]] int smask = 3;
        if constexpr (kSum && !kCoarse) {
          // SUM_THRESH: every cell was decided above (sum_near for the ones
          // near the threshold); the exact path is not needed
          trig = false;
          smask = 0;
        }
        if constexpr (kBound) {
          // no candidates
        } else if constexpr (kSum && !kCoarse) {
          // A step of a pair whose first step is pending joins that pending
          // two-step block (its segments in mask bits 2, 3); others queue in
          // rank order while there is room, else become the pending step.
          // (The sums must not walk a segment twice.)
          const bool want_q = trig && pend < 0;
          if (trig && pend >= 0) pmsk |= smask << 2;
          const unsigned tmask = __ballot_sync(0xffffffffu, want_q);
          if (tmask) {
            const int rank = __popc(tmask & ((1u << lane) - 1u));
            if (want_q) {
              if (qn + rank < kQueue) {
                SlowItem& it = sm.queue[warp][qn + rank];
#pragma unroll
                for (int k = 0; k < kDiags; ++k) it.cov[k] = cov[k];
                it.vw = make_float2(vx, vy);
                it.s = s | (1 << 8) | (smask << 16);
                it.owner = t;
              } else {
                pend = s;
                pmsk = smask;
              }
            }
            const int nq = qn + __popc(tmask);
            qn = nq < kQueue ? nq : kQueue;
          }
          n_slow += trig ? 1u : 0u;
        } else {
          // queue the triggered lanes in rank order while there is room;
          // the exact path walks both segments of every step of the block
          // (a cell of 1NN_INDEX published twice changes nothing)
          const unsigned tmask = __ballot_sync(0xffffffffu, trig);
          if (tmask) {
            const int rank = __popc(tmask & ((1u << lane) - 1u));
            if (trig) {
              if (qn + rank < kQueue) {
                SlowItem& it = sm.queue[warp][qn + rank];
#pragma unroll
                for (int k = 0; k < kDiags; ++k) it.cov[k] = cov[k];
                it.vw = make_float2(vx, vy);
                it.s = s | (1 << 8) | (15 << 16);
                it.owner = t;
              } else if (pend < 0) {
                pend = s;
              }
            }
            const int nq = qn + __popc(tmask);
            qn = nq < kQueue ? nq : kQueue;
            n_slow += trig ? 1u : 0u;
          }
        }
        if constexpr (kExact) {
          // the bound of a block that starts in the pair's first step: E at
          // its end plus both steps' roundings for the steps back
          vlast = P == 0 ? dE : make_float2(vx + vlast.x, vy + vlast.y);
        } else {
          vlast = make_float2(vx, vy);
        }
      };
#pragma unroll 1
      for (int s = 0; s < nsteps; s += 2) {
        {
          const int rb = (rq + s + t) < kBlocks ? (rq + s + t) : (rq + s + t - kBlocks);
          if constexpr (kWindow) {
#pragma unroll
            for (int x = 0; x < kDiags - 1; ++x) {
              cfw[x] = col_fg(sm, 9 * rb + x);  // padc(ring column 8 rb + x), x < 8
              if constexpr (!kCoarse) ciw[x] = sm.u.s.c_iv[9 * rb + x];
            }
          }
        }
        step(s, Parity<0>());
        step(s + 1, Parity<1>());
        if constexpr (kBound) continue;
        // between pairs: drain a half-full queue (every queue at the slab's
        // end), then queue and drain the steps that found it full
        const unsigned pmask = __ballot_sync(0xffffffffu, pend >= 0);
        if (pmask || qn >= kQueue / 2 || (qn && s + 2 == nsteps)) {
          if (qn) {
            n_verify += kExact ? drain_exact<kMat>(sm, warp, qn, lane)
                               : drain_queue<!kCoarse>(sm, warp, qn, lane);
            qn = 0;
          }
          const int np = __popc(pmask);
          const int rank = __popc(pmask & ((1u << lane) - 1u));
          for (int done = 0; done < np; done += kQueue) {
            if (pend >= 0 && rank >= done && rank < done + kQueue) {
              SlowItem& it = sm.queue[warp][rank - done];
#pragma unroll
              for (int k = 0; k < kDiags; ++k) it.cov[k] = cov[k];
              it.vw = vlast;
              it.s = pend | ((s + 2 - pend) << 8) | (pmsk << 16);
              it.owner = t;
            }
            const int take = (np - done) < kQueue ? (np - done) : kQueue;
            n_verify += kExact ? drain_exact<kMat>(sm, warp, take, lane)
                               : drain_queue<!kCoarse>(sm, warp, take, lane);
          }
          pend = -1;
        }
      }
      if constexpr (kRaise) {
        // the columns after the last step's first 8
        const int rb = (rq + nsteps + t) < kBlocks ? (rq + nsteps + t) : (rq + nsteps + t - kBlocks);
#pragma unroll
        for (int x = 0; x < kDiags - 1; ++x)
          raise_shared(sm.c_best[9 * rb + x], __float_as_uint(cnext[x].x), __float_as_uint(cnext[x].y));
        __syncthreads();
        const float2 v = sm.r_best[t];
        raise_bound(pr.key_row, rbase[0] + t, v.x, P.kl, P.knn_k);
        raise_bound(pr.key_row, rbase[1] + t, v.y, P.kl, P.knn_k);
        if (q + 1 == nslabs) {
          for (int c = t; c < ncols; c += kThreads) {
            const float2 u = sm.c_best[padc(ringc(ring0, c))];
            raise_bound(pr.key_col, cbase_g[0] + c, u.x, P.kl, P.knn_k);
            raise_bound(pr.key_col, cbase_g[1] + c, u.y, P.kl, P.knn_k);
          }
          __syncthreads();  // sm.prob is read above
        }
        continue;
      }
      n_steps += nsteps;
      __syncthreads();
      if constexpr (kExact && !kBound) {
        // A unit whose cells its FP32 values cannot rule out (error bounds
        // above the spread of the correlations: near-flat windows beside
        // large steps, exact repeats everywhere) is left to the FP64 band
        // kernel; what it published stands.
        const bool leave = sm.cx.unit_lost;
        __syncthreads();
        if (leave) {
          if (t == 0) {
            P.fp64_list[atomicAdd(P.fp64_count, 1ull)] = u;
            P.fp64_unit[u] = 1;
          }
          break;
        }
      }
      if (sum_mode && pr.sum_row) {
        // the slab's row sums (thread t: row t; it restages row t next)
        const float2 v = sm.r_best[t];
        const int64_t i0 = rbase[0] + t, i1 = rbase[1] + t;
        if (v.x != 0.f && i0 < rend[0]) atomicAdd(pr.sum_row + i0, static_cast<double>(v.x));
        if (v.y != 0.f && i1 < rend[1]) atomicAdd(pr.sum_row + i1, static_cast<double>(v.y));
      }
      if (sum_mode && pr.sum_col && q + 1 == nslabs) {
        // unit end: every column left in the ring
        for (int c = t; c < ncols; c += kThreads) {
          const float2 v = sm.c_best[padc(ringc(ring0, c))];
          const int64_t j0 = cbase_g[0] + c, j1 = cbase_g[1] + c;
          if (v.x != 0.f && j0 < pr.C.ns) atomicAdd(pr.sum_col + j0, static_cast<double>(v.x));
          if (v.y != 0.f && j1 < pr.C.ns) atomicAdd(pr.sum_col + j1, static_cast<double>(v.y));
        }
      }
      // The flushes read the unit's Problem in shared memory, which thread 0
      // overwrites when it fetches the next unit.
      if (sum_mode && q + 1 == nslabs) __syncthreads();
    }
  }
  if constexpr (!kBound && !kRuns) {
    __syncwarp();
    sm.cx.vcap = P.vreq_cap;  // (a CTA without a unit has no context; every writer the same)
    sm.cx.vreq = P.vreq;
    close_requests(sm, sm.cx, warp, lane);
  }
  // per-CTA totals of the work counters
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    n_steps += __shfl_xor_sync(0xffffffffu, n_steps, o);
    n_slow += __shfl_xor_sync(0xffffffffu, n_slow, o);
    n_verify += __shfl_xor_sync(0xffffffffu, n_verify, o);
  }
  if (lane == 0 && P.counters) {
    atomicAdd(P.counters + 0, n_steps);
    atomicAdd(P.counters + 1, n_slow);
    atomicAdd(P.counters + 2, n_verify);
  }
  if constexpr (kRuns) {
#pragma unroll
    for (int g = 0; g < 2; ++g)
#pragma unroll
      for (int h = 0; h < 2; ++h)
        if (mrun.cell[g][h] >= 0) atomicMax(P.mat + mrun.cell[g][h], ord_float(mrun.mx[g][h]));
  }
  if constexpr (kSum || (kMat && !kExact)) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) tfast = fmaxf(tfast, __shfl_xor_sync(0xffffffffu, tfast, o));
    if (lane == 0 && P.counters && tfast > 0.f)
      atomicMax(P.counters + 4, static_cast<unsigned long long>(__float_as_uint(tfast)));
  }
}

}  // namespace

size_t mixed_1nn_smem_bytes() { return sizeof(Smem); }

__global__ void __launch_bounds__(kThreads, 4) join_mixed_1nn_kernel(JoinParams P) {
  band_body<false, false>(P);
}

// (three CTAs per SM: with the registers of four, 220 bytes spilled per
// thread; 200003 samples, m = 256, r > 0.5 18.8 -> 17.6 ms, m = 100, r > 0.9
// 15.1 -> 13.3)
__global__ void __launch_bounds__(kThreads, 3) join_mixed_sum_kernel(JoinParams P) {
  band_body<true, false>(P);
}

__global__ void __launch_bounds__(kThreads, 4) join_mixed_mat_kernel(JoinParams P) {
  band_body<false, false, true>(P);
}

__global__ void __launch_bounds__(kThreads, 4) join_mixed_knn_kernel(JoinParams P) {
  band_body<false, false, false, true>(P);
}

__global__ void __launch_bounds__(kThreads, 4) join_mixed_1nn_coarse_kernel(JoinParams P) {
  band_body<false, true>(P);
}

__global__ void __launch_bounds__(kThreads, 4) join_mixed_sum_coarse_kernel(JoinParams P) {
  band_body<true, true>(P);
}

__global__ void __launch_bounds__(kThreads, 4) join_exact_1nn_kernel(JoinParams P) {
  band_body<false, false, false, false, true>(P);
}

__global__ void __launch_bounds__(kThreads, 4) bound_exact_1nn_kernel(JoinParams P) {
  band_body<false, false, false, false, true, true>(P);
}

__global__ void __launch_bounds__(kThreads, 4) join_exact_mat_kernel(JoinParams P) {
  band_body<false, false, true, false, true>(P);
}

__global__ void __launch_bounds__(kThreads, 4) bound_exact_mat_kernel(JoinParams P) {
  band_body<false, false, true, false, true, true>(P);
}

__global__ void knn_floor_kernel(const unsigned long long* __restrict__ bounds,
                                 const unsigned long long* __restrict__ lists, int64_t n, int k,
                                 double thr, KeyLayout kl, uint64_t* __restrict__ out) {
  const int64_t w = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
  if (w >= n) return;
  const uint64_t a = bounds[w * k + k - 1] >> kl.idx_bits, b = lists[w * k + k - 1] >> kl.idx_bits;
  const uint64_t c = q_from_float_bits(__float_as_uint(__double2float_rd(thr)), kl.frac_bits);
  const uint64_t q = a > b ? (a > c ? a : c) : (b > c ? b : c);
  out[w] = q << kl.idx_bits;
}

// Settles the verification requests of the band kernels, one warp per
// cell.  A request whose upper bound rv + margin no longer exceeds the
// current best of its row or column cannot change the profile and is
// skipped; otherwise the cell's covariance is computed directly from the
// FP32 series copies (each factor centred per window) and its r merged into
// both profiles.  Runs after the join on the same stream; the request count
// is read on the device.
__global__ void __launch_bounds__(256)
verify_requests_kernel(JoinParams P) {
  const int lane = threadIdx.x & 31;
  const unsigned long long total = P.counters[3];
  const int64_t n = total < static_cast<unsigned long long>(P.vreq_cap)
                        ? static_cast<int64_t>(total) : P.vreq_cap;
  // A block takes kReqChunk requests in a row, what one warp of the join
  // wrote: cells of neighbouring windows, whose samples its warps share in L1
  // (one dot of m = 1024 reads 8 KB, from L2 the kernel's bound: 9.3e6
  // requests 10.9 -> 8.9 ms, 2^18 x 2^17 windows of m = 256 0.91 -> 0.79 ms)
  const int nwarps = blockDim.x >> 5;
  for (int64_t w0 = static_cast<int64_t>(blockIdx.x) * kReqChunk; w0 < n;
       w0 += static_cast<int64_t>(gridDim.x) * kReqChunk)
  for (int64_t w = w0 + (threadIdx.x >> 5); w < w0 + kReqChunk && w < n; w += nwarps) {
    const VerifyReq rq = P.vreq[w];
    const Problem& pr = problem_of(P, static_cast<int>(rq.i >> 40));
    const int64_t i = static_cast<int64_t>(rq.i & ((uint64_t{1} << 40) - 1));
    const int64_t j = i + rq.d;
    if (P.profile_type == 2) {  // SUM_THRESH: the cell counts if above it
      if (rq.ub < -3.f) continue;  // an unused slot
      const float cv = verify_cov_warp(pr.R, pr.C, i, j, pr.m, lane);
      const float rv = (cv * pr.C.inv32[j]) * pr.R.inv32[i];
      if (lane == 0 && rv > static_cast<float>(P.threshold)) {
        if (pr.sum_row) atomicAdd(pr.sum_row + i, static_cast<double>(rv));
        if (pr.sum_col) atomicAdd(pr.sum_col + j, static_cast<double>(rv));
      }
      continue;
    }
    if (P.knn_k > 0) {  // APPROX_ALL_NEIGHBORS: into the k-best lists
      const int k = P.knn_k;
      const float thr = static_cast<float>(P.threshold);
      // decided by lane 0 for the warp: the lists change under other
      // warps' (and lane 0's own) atomics, and the lanes' loads of them need
      // not agree, while the shuffles of the dot need every lane
      bool ro = pr.key_row && rq.ub > knn_floor(pr.key_row + i * k, k, thr, P.kl);
      bool co = pr.key_col && rq.ub > knn_floor(pr.key_col + j * k, k, thr, P.kl);
      ro = __shfl_sync(0xffffffffu, ro, 0);
      co = __shfl_sync(0xffffffffu, co, 0);
      if (!ro && !co) continue;
      const float cv = verify_cov_warp(pr.R, pr.C, i, j, pr.m, lane);
      if (lane == 0) {
        const float rv = (cv * pr.C.inv32[j]) * pr.R.inv32[i];
        if (rv > thr) {
          const uint64_t q = q_from_float_bits(__float_as_uint(rv), P.kl.frac_bits);
          if (ro && rv > knn_floor(pr.key_row + i * k, k, thr, P.kl))
            topk_insert(reinterpret_cast<u64*>(pr.key_row + i * k), k, make_key(q, j, P.kl));
          if (co && rv > knn_floor(pr.key_col + j * k, k, thr, P.kl))
            topk_insert(reinterpret_cast<u64*>(pr.key_col + j * k), k, make_key(q, i, P.kl));
        }
      }
      continue;
    }
    // warp-uniform by lane 0's view, as above
    bool row_open = pr.key_row && rq.ub > key_corr_floor(pr.key_row[i], P.kl);
    bool col_open = pr.key_col && rq.ub > key_corr_floor(pr.key_col[j], P.kl);
    row_open = __shfl_sync(0xffffffffu, row_open, 0);
    col_open = __shfl_sync(0xffffffffu, col_open, 0);
    if (!row_open && !col_open) continue;
    const float cv = verify_cov_warp(pr.R, pr.C, i, j, pr.m, lane);
    if (lane == 0) {
      const float rv = (cv * pr.C.inv32[j]) * pr.R.inv32[i];
      const uint64_t q = q_from_float_bits(__float_as_uint(rv), P.kl.frac_bits);
      if (row_open) atomicMax(reinterpret_cast<u64*>(pr.key_row + i), make_key(q, j, P.kl));
      if (col_open) atomicMax(reinterpret_cast<u64*>(pr.key_col + j), make_key(q, i, P.kl));
    }
  }
}

// ---------------------------------------------------------------------------
// Seeds of the mixed 1NN join (an approximate pre-pass in the manner of
// SCRIMP++'s PreSCRIMP).  A join of the series averaged over blocks of f
// samples (window m / f) gives every block-averaged window a likely partner;
// each full-resolution window i = f i' + o then gets the exact correlation of
// the cell on the same diagonal, (i, f idx(i') + o), merged into the profile
// keys before the band kernel runs.  Every seed is a real cell's r, so the
// join's result is unchanged; its filters simply start high, which spares
// most of the exact-path work of the first bands.
// ---------------------------------------------------------------------------

// out[k] = mean of T[f k .. f k + f), NaN when any of them is not finite.
__global__ void paa_kernel(const double* __restrict__ T, int64_t n_out, int f,
                           double* __restrict__ out) {
  const int64_t k = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
  if (k >= n_out) return;
  double sum = 0.0;
  bool finite = true;
  for (int u = 0; u < f; ++u) {
    const double v = T[static_cast<int64_t>(f) * k + u];
    finite = finite && isfinite(v);
    sum += v;
  }
  out[k] = finite ? sum / f : __longlong_as_double(0x7FF8000000000000ll);
}

// Packed entries {r = floor, index 0}: the pre-pass only looks for partners
// above `floor`, which spares it the cold start of a join from "no match".
__global__ void fill_floor_kernel(uint64_t* __restrict__ p, int64_t n, float floor) {
  const int64_t k = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
  if (k < n) p[k] = __float_as_uint(floor);
}

// One warp per window i of X: its seed partner from the block-averaged
// profile, the exact r of that cell, merged into X's keys (and Y's).
__global__ void __launch_bounds__(256) seed_kernel(SeedArgs S) {
  const int lane = threadIdx.x & 31;
  const int64_t nwarps = static_cast<int64_t>(gridDim.x) * (blockDim.x >> 5);
  for (int64_t i = (static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x) >> 5;
       i < S.X.ns; i += nwarps) {
    const int64_t ib = i / S.factor;
    const int64_t ip = ib < S.ns_paa ? ib : S.ns_paa - 1;
    const uint64_t packed = S.paa[ip];
    if (!(__uint_as_float(static_cast<uint32_t>(packed)) > S.floor)) continue;  // no partner found
    const int64_t j = S.factor * static_cast<int64_t>(packed >> 32) + (i - S.factor * ip);
    if (j >= S.Y.ns) continue;
    if (S.excl >= 0 && (j - i < S.excl && i - j < S.excl)) continue;  // trivial match
    const float ivx = S.X.inv32[i], ivy = S.Y.inv32[j];
    if (isnan(ivx) || isnan(ivy)) continue;
    const float cv = verify_cov_warp(S.X, S.Y, i, j, S.m, lane);
    if (lane == 0) {
      const uint64_t q = q_from_float_bits(__float_as_uint((cv * ivy) * ivx), S.kl.frac_bits);
      atomicMax(reinterpret_cast<u64*>(S.key_x + i), make_key(q, j, S.kl));
      if (S.key_y) atomicMax(reinterpret_cast<u64*>(S.key_y + j), make_key(q, i, S.kl));
    }
  }
}

// Seeds of self-joins from diagonals near the exclusion zone, one thread per
// window: cells (i, i + d_lo + 16 s), s < kDiagSeeds, are real cells of the
// join, so their r are valid starting bests for window i (as a row) and the
// partner windows (as columns).  Where the series moves slowly against the
// window length (random walks) they are close to the final bests, and the
// filter starts high instead of sending every block of the first slabs to
// the exact path.  win_prefix[p] is the first global window of problem p.
constexpr int kDiagSeeds = 8;
constexpr int kDiagSeedStep = 16;
__global__ void __launch_bounds__(256) diag_seed_kernel(const Problem* __restrict__ probs,
                                                        const int64_t* __restrict__ win_prefix,
                                                        int nprob, KeyLayout kl) {
  const int64_t total = win_prefix[nprob];
  const int64_t stride = static_cast<int64_t>(gridDim.x) * blockDim.x;
  for (int64_t w = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; w < total;
       w += stride) {
    int lo = 0, hi = nprob;
    while (hi - lo > 1) {
      const int mid = (lo + hi) >> 1;
      if (win_prefix[mid] <= w) lo = mid; else hi = mid;
    }
    const Problem& pr = probs[lo];
    const int64_t i = w - win_prefix[lo];
    if (i >= pr.R.ns) continue;
    const float ivx = pr.R.inv32[i];
    if (isnan(ivx)) continue;
    uint64_t best = 0;
    for (int s = 0; s < kDiagSeeds; ++s) {
      const int64_t j = i + pr.d_lo + static_cast<int64_t>(s) * kDiagSeedStep;
      if (j >= pr.C.ns) break;
      const float ivy = pr.C.inv32[j];
      if (isnan(ivy)) continue;
      const float cv = verify_cov_lane(pr.R, pr.C, i, j, pr.m);
      const uint64_t q = q_from_float_bits(__float_as_uint((cv * ivy) * ivx), kl.frac_bits);
      if (pr.key_col) atomicMax(reinterpret_cast<u64*>(pr.key_col + j), make_key(q, i, kl));
      const uint64_t kr = make_key(q, j, kl);
      best = kr > best ? kr : best;
    }
    if (pr.key_row && best) atomicMax(reinterpret_cast<u64*>(pr.key_row + i), best);
  }
}

// Largest p with prefix[p] <= t (prefix[0] = 0, p < n).
__device__ __forceinline__ int job_of(const int64_t* __restrict__ prefix, int n, int64_t t) {
  int lo = 0, hi = n;
  while (hi - lo > 1) {
    const int mid = (lo + hi) >> 1;
    if (prefix[mid] <= t) lo = mid; else hi = mid;
  }
  return lo;
}

__global__ void paa_batch_kernel(const PaaJob* __restrict__ jobs,
                                 const int64_t* __restrict__ out_prefix, int njobs) {
  const int64_t total = out_prefix[njobs];
  const int64_t stride = static_cast<int64_t>(gridDim.x) * blockDim.x;
  for (int64_t t = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; t < total;
       t += stride) {
    const int p = job_of(out_prefix, njobs, t);
    const PaaJob& J = jobs[p];
    const int64_t k = t - out_prefix[p];
    double sum = 0.0;
    bool finite = true;
    for (int u = 0; u < J.f; ++u) {
      const double v = J.src[static_cast<int64_t>(J.f) * k + u];
      finite = finite && isfinite(v);
      sum += v;
    }
    J.dst[k] = finite ? sum / J.f : __longlong_as_double(0x7FF8000000000000ll);
  }
}

__global__ void fill_key_floor_kernel(uint64_t* __restrict__ keys, int64_t n, float floor,
                                      KeyLayout kl) {
  const uint64_t key = make_key(q_from_float_bits(__float_as_uint(floor), kl.frac_bits), 0, kl);
  const int64_t stride = static_cast<int64_t>(gridDim.x) * blockDim.x;
  for (int64_t k = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; k < n; k += stride)
    keys[k] = key;
}

// One warp per block-averaged window i' of a series (PreSCRIMP-style seeds
// with a neighbourhood refinement): its pre-pass partner j' puts the windows
// i = f i' + o (o < f) near diagonal D = f (j' - i'); lane l takes diagonal
// D + l - 15 (|l - 15| < f), computes its first cell's covariance directly
// (FP32, centred) and walks the block's rows with the FP32 recurrence; per
// row the warp keeps the best of its cells, merged into that window's key.
// Every seed is a real cell's r, so the join's result does not depend on
// them; good seeds only spare the join's exact path the records a cold start
// sets (a short series' best improves about ln(n) times as the bands sweep
// outward).
__global__ void __launch_bounds__(256) batch_seed_kernel(const BatchSeedJob* __restrict__ jobs,
                                                         const int64_t* __restrict__ paa_prefix,
                                                         int njobs, KeyLayout kl, float floor) {
  const int lane = threadIdx.x & 31;
  const int64_t total = paa_prefix[njobs];
  const int64_t nwarps = static_cast<int64_t>(gridDim.x) * (blockDim.x >> 5);
  const uint64_t q_floor = q_from_float_bits(__float_as_uint(floor), kl.frac_bits);
  for (int64_t w = (static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x) >> 5; w < total;
       w += nwarps) {
    const int p = job_of(paa_prefix, njobs, w);
    const BatchSeedJob& J = jobs[p];
    const int64_t ip = w - paa_prefix[p];
    const uint64_t pk = J.paa_key[ip];
    if ((pk >> kl.idx_bits) <= q_floor) continue;  // no partner above the floor (warp-uniform)
    const int64_t jp = static_cast<int64_t>(kl.idx_mask - (pk & kl.idx_mask));
    const int f = J.f;
    const int64_t ns = J.X.ns;
    const int64_t i0 = static_cast<int64_t>(f) * ip;
    const int delta = lane - 15;
    const int64_t d = static_cast<int64_t>(f) * (jp - ip) + delta;
    // rows o in [o_lo, o_hi) of this lane's diagonal are cells of the join
    int64_t o_lo = 0, o_hi = 0;
    if (lane < 31 && (delta < f && -delta < f) && (d >= J.excl || -d >= J.excl)) {
      o_lo = -(i0 + d) > 0 ? -(i0 + d) : 0;
      o_hi = f;
      if (ns - i0 < o_hi) o_hi = ns - i0;
      if (ns - i0 - d < o_hi) o_hi = ns - i0 - d;
    }
    float cov = 0.f;
    if (o_lo < o_hi) cov = cov_part(J.X, J.X, i0 + o_lo, i0 + o_lo + d, 0, J.m);
    for (int o = 0; o < f; ++o) {
      const int64_t i = i0 + o, j = i + d;
      const bool valid = o >= o_lo && o < o_hi;
      uint64_t key = 0;
      if (valid) {
        const float ivi = J.X.inv32[i], ivj = J.X.inv32[j];
        if (!isnan(ivi) && !isnan(ivj))
          key = make_key(q_from_float_bits(__float_as_uint((cov * ivj) * ivi), kl.frac_bits), j, kl);
        if (o + 1 < o_hi)
          cov = fmaf(J.X.df32[i], J.X.dg32[j], fmaf(J.X.df32[j], J.X.dg32[i], cov));
      }
#pragma unroll
      for (int s = 16; s > 0; s >>= 1) {
        const uint64_t other = __shfl_xor_sync(0xffffffffu, key, s);
        key = other > key ? other : key;
      }
      if (lane == 0 && key && i < ns) atomicMax(reinterpret_cast<u64*>(J.key + i), key);
    }
  }
}

int mixed_1nn_band_width() { return kBand; }
int mixed_1nn_slab_rows() { return kSlab; }
int mixed_1nn_threads() { return kThreads; }

}  // namespace scamp_gb300
