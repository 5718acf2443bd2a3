// final_eval.cu -- cells evaluated directly in FP64: the re-evaluation of
// every reported 1NN cell, and the requests of the double-precision joins that
// run behind the FP32 filter.
//
// Both join forms choose each window's best partner from a recurrence (FP64
// in the plain form, FP32 behind a filter in the others).  Before the
// profile is written back, this kernel recomputes the correlation of every
// (window, reported partner) pair directly: the centred FP64 dot product
// times the two windows' inverse norms (stats.cu: compensated sums of
// squares), so the value a join reports does not carry the recurrence's
// drift.  This is the reference's correlation formula
// (src/cpu_kernels.cpp:166-171 with the norms of src/cpu_stats.cpp:85-97)
// evaluated once per reported cell.  Bound by the FP64 pipe at 3 operations
// per sample (with the sums of squares formed again for every pair, 5:
// 2^20 windows of m = 1024 9.8 -> 6.0 ms).
//
// Error bound (per reported value, against the exact correlation of the two
// FP64 windows), u = 2^-53, gamma_k = k u / (1 - k u): every centred term
// x_t = fl(T - mu) carries one rounding; each of a group's 8 lanes sums its
// terms by FMA into two accumulators of at most ceil(m / 16) terms, one add
// joins them and three shuffle levels add the lanes' sums, so the dot is off
// by gamma_{ceil(m/16) + 6} ||x|| ||y||; an inverse norm by 5 u at
// most (its sum of squares is compensated throughout, and summed directly where
// the recurrence's residue could show; then its rounding, a square root and a
// quotient); two products follow.  (The means' own rounding adds m times the
// product of two of them, second order: it shows where a series' offset is 10^8
// and more times its windows' deviation.)
// Together at most gamma_{ceil(m/16) + 18}, within the stated
//   |r_hat - r| <= 2 gamma_{ceil(m/16) + 10}.
// The 64-bit key then keeps r to 2^-F.  The host adds the two
// (final_eval_bound).
//
// Entries the join did not change (a best-so-far entry given on input, whose
// index may refer to another join) are left as they are.
#include <cstdint>

#include "engine.cuh"

namespace scamp_gb300 {

namespace {

constexpr int kLanes = 8;  // lanes per window: four windows per warp

// Direct FP64 covariance of window i of X with window j of Y by kLanes lanes,
// times the two windows' inverse norms; valid in every lane of the group.
__device__ __forceinline__ double corr_group_norms(const SeriesDev& X, const SeriesDev& Y,
                                                   int64_t i, int64_t j, int64_t m, int sub) {
  const double mx = X.mean[i], my = Y.mean[j];
  const double* __restrict__ tx = X.T + i;
  const double* __restrict__ ty = Y.T + j;
  double s0 = 0.0, s1 = 0.0;
  int64_t t = sub;
  for (; t + kLanes < m; t += 2 * kLanes) {
    s0 = fma(tx[t] - mx, ty[t] - my, s0);
    s1 = fma(tx[t + kLanes] - mx, ty[t + kLanes] - my, s1);
  }
  if (t < m) s0 = fma(tx[t] - mx, ty[t] - my, s0);
  s0 += s1;
#pragma unroll
  for (int o = kLanes / 2; o > 0; o >>= 1) s0 += __shfl_xor_sync(0xffffffffu, s0, o);
  return s0 * Y.inv[j] * X.inv[i];
}

__device__ __forceinline__ uint64_t corr_key(double r, int64_t index, const KeyLayout& kl) {
  return make_key(q_from_double_bits(__double_as_longlong(r), kl.frac_bits), index, kl);
}

// The key an input profile entry turns into (profile_to_keys_kernel,
// floats_to_keys_kernel): 0 when there is no entry.
__device__ __forceinline__ uint64_t initial_key(const EvalSide& s, int64_t w, const KeyLayout& kl) {
  if (s.prof_in) {
    const uint64_t e = s.prof_in[w];
    const uint32_t cbits = static_cast<uint32_t>(e);
    const uint32_t idx = static_cast<uint32_t>(e >> 32);
    if (!(__uint_as_float(cbits) >= -1.0f) || static_cast<uint64_t>(idx) > kl.idx_mask) return 0;
    return make_key(q_from_float_bits(cbits, kl.frac_bits), idx, kl);
  }
  if (s.max_in) {
    const float c = s.max_in[w];
    if (!(c >= -1.0f)) return 0;
    return make_key(q_from_float_bits(__float_as_uint(c), kl.frac_bits), 0, kl);
  }
  return 0;
}

// Window w of side s, evaluated by the kLanes lanes of group `sub`; every
// lane of the warp calls it (the shuffle tree needs them), `active` marks the
// groups with a window.
__device__ __forceinline__ void eval_window(const EvalSide& s, int64_t w, int64_t m,
                                            const KeyLayout& kl, int sub, bool active) {
  uint64_t k = active ? s.keys[w] : 0;
  if (k != 0 && k == initial_key(s, w, kl)) k = 0;
  int64_t j = k ? key_to_index(k, kl) : 0;
  if (j < 0 || j >= s.Y.ns) k = 0;
  // groups with nothing to do still take part in the shuffles (no terms)
  const bool work = k != 0;
  const double r = corr_group_norms(s.X, s.Y, work ? w : 0, work ? j : 0, work ? m : 0, sub);
  if (sub == 0 && work && !isnan(r)) {
    // |r| <= 1 up to rounding; the key holds r in [-2, 2)
    const double rc = r > 1.0 ? 1.0 : (r < -1.0 ? -1.0 : r);
    s.keys[w] = make_key(q_from_double_bits(__double_as_longlong(rc), kl.frac_bits), j, kl);
  }
}

// The key entry `e` of an input k-best list turns into: 0 when empty.
__device__ __forceinline__ uint64_t list_entry_key(uint64_t e, const KeyLayout& kl) {
  const uint32_t cbits = static_cast<uint32_t>(e);
  const uint32_t idx = static_cast<uint32_t>(e >> 32);
  if (!(__uint_as_float(cbits) >= -1.0f) || static_cast<uint64_t>(idx) > kl.idx_mask) return 0;
  return make_key(q_from_float_bits(cbits, kl.frac_bits), idx, kl);
}

constexpr int kKnnMaxK = 64;  // longest list the mixed k-best form keeps

}  // namespace

int knn_mixed_max_k() { return kKnnMaxK; }

// k-best lists: kLanes lanes per window, its k entries in turn (the slot loop
// is warp-uniform, so the shuffle tree always has its lanes), then the
// group's first lane re-sorts the list, largest key first (ties: the smaller
// index, which the key's index field orders first).
__global__ void __launch_bounds__(256) knn_final_eval_kernel(EvalSide S, int k, double thr,
                                                             KeyLayout kl) {
  const int lane = threadIdx.x & 31;
  const int sub = lane & (kLanes - 1);
  const int64_t nwarps = static_cast<int64_t>(gridDim.x) * (blockDim.x >> 5);
  constexpr int kGroups = 32 / kLanes;
  for (int64_t g0 = ((static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x) >> 5) * kGroups;
       g0 < S.ns; g0 += nwarps * kGroups) {
    const int64_t w = g0 + lane / kLanes;
    const bool active = w < S.ns;
    uint64_t* list = S.keys + (active ? w : 0) * k;
    for (int s = 0; s < k; ++s) {
      uint64_t key = active ? list[s] : 0;
      if (key != 0 && S.prof_in) {
        // an entry of the given list stays as it is
        for (int t = 0; t < k; ++t)
          if (list_entry_key(S.prof_in[w * k + t], kl) == key) {
            key = 0;
            break;
          }
      }
      const int64_t j = key ? key_to_index(key, kl) : 0;
      const bool work = key != 0 && j >= 0 && j < S.Y.ns;
      const double r = corr_group_norms(S.X, S.Y, work ? w : 0, work ? j : 0, work ? S.m : 0, sub);
      if (sub == 0 && work) {
        const double rc = r > 1.0 ? 1.0 : (r < -1.0 ? -1.0 : r);
        list[s] = (!isnan(r) && r > thr)
                      ? make_key(q_from_double_bits(__double_as_longlong(rc), kl.frac_bits), j, kl)
                      : 0;
      }
    }
    if (sub == 0 && active) {
      uint64_t v[kKnnMaxK];
      const int kc = k < kKnnMaxK ? k : kKnnMaxK;
      for (int s = 0; s < kc; ++s) {
        const uint64_t x = list[s];
        int p = s;
        while (p > 0 && v[p - 1] < x) {
          v[p] = v[p - 1];
          --p;
        }
        v[p] = x;
      }
      for (int s = 0; s < kc; ++s) list[s] = v[s];
    }
  }
}

// Settles the exact form's requests: every cell that may count gets its FP64
// r and enters its row's and its column's results: the best (1NN), the k-best
// lists (knn_k > 0) or the grid (mat).  A request whose upper bound the
// results have meanwhile reached is skipped (decided by the group's first
// lane: the lanes' loads need not agree), and so is one of a unit left to the
// FP64 kernels, which have entered its cells (a list would hold them twice).
__global__ void __launch_bounds__(256) verify_exact_kernel(JoinParams P) {
  const int lane = threadIdx.x & 31;
  const int sub = lane & (kLanes - 1);
  const unsigned long long total = P.counters[3];
  const int64_t n = total < static_cast<unsigned long long>(P.vreq_cap)
                        ? static_cast<int64_t>(total) : P.vreq_cap;
  constexpr int kGroups = 32 / kLanes;
  const int k = P.knn_k;
  const bool plain = k == 0 && !P.mat;
  const bool some_left = *P.fp64_count > 0;
  const float thr = plain ? -3.f : __double2float_rd(P.threshold);
  // a block takes 64 requests in a row (verify_requests_kernel)
  constexpr int kRun = 64;
  const int step = (blockDim.x >> 5) * kGroups;
  for (int64_t run = static_cast<int64_t>(blockIdx.x) * kRun; run < n;
       run += static_cast<int64_t>(gridDim.x) * kRun)
  for (int64_t g0 = run + (threadIdx.x >> 5) * kGroups; g0 < run + kRun && g0 < n; g0 += step) {
    const int64_t g = g0 + lane / kLanes;
    const VerifyReq rq = P.vreq[g < n ? g : g0];
    const int p = static_cast<int>(rq.i >> 40);
    const Problem& pr = P.prob[p];
    const int64_t i = static_cast<int64_t>(rq.i & ((uint64_t{1} << 40) - 1));
    const int64_t j = i + rq.d;
    bool row, col;
    unsigned *er = nullptr, *ec = nullptr;  // the cell's grid entries
    if (P.mat) {
      if (P.mat_col[p]) ec = P.mat + div_magic(i, P.rpc_magic) * P.mat_w + div_magic(j, P.cpc_magic);
      if (P.mat_row[p]) er = P.mat + div_magic(j, P.rpc_magic) * P.mat_w + div_magic(i, P.cpc_magic);
      // (>=: an entry rounded to a float may lie above its FP64 value)
      row = er && rq.ub >= float_of_ord(__ldcg(er));
      col = ec && rq.ub >= float_of_ord(__ldcg(ec));
    } else {
      row = pr.key_row && rq.ub > key_corr_floor(__ldcg(pr.key_row + (k ? i * k + k - 1 : i)), P.kl);
      col = pr.key_col && rq.ub > key_corr_floor(__ldcg(pr.key_col + (k ? j * k + k - 1 : j)), P.kl);
    }
    bool counts = g < n && rq.ub > thr;
    if (some_left && counts) {
      const int64_t band = (static_cast<int64_t>(rq.d) - pr.d_lo) / P.band_width;
      counts = !P.fp64_unit[P.band_unit_prefix[pr.band_begin + band] + i / (2 * P.seg_len)];
    }
    row = row && counts;
    col = col && counts;
    const unsigned open = __ballot_sync(0xffffffffu, sub == 0 && (row || col));
    if (!open) continue;
    const bool work = (open >> (lane & ~(kLanes - 1))) & 1u;
    const double r = corr_group_norms(pr.R, pr.C, i, j, work ? P.m : 0, sub);
    if (sub != 0 || !work || isnan(r) || !(plain || r > P.threshold)) continue;
    if (P.mat) {
      const unsigned v = ord_float(static_cast<float>(r));
      if (row) atomicMax(er, v);
      if (col) atomicMax(ec, v);
    } else if (k) {
      unsigned long long* lr = reinterpret_cast<unsigned long long*>(pr.key_row + i * k);
      unsigned long long* lc = reinterpret_cast<unsigned long long*>(pr.key_col + j * k);
      const uint64_t kr = corr_key(r, j, P.kl), kc = corr_key(r, i, P.kl);
      if (row && kr > __ldcg(lr + k - 1)) topk_insert(lr, k, kr);
      if (col && kc > __ldcg(lc + k - 1)) topk_insert(lc, k, kc);
    } else {
      if (row) atomicMax(reinterpret_cast<unsigned long long*>(pr.key_row + i), corr_key(r, j, P.kl));
      if (col) atomicMax(reinterpret_cast<unsigned long long*>(pr.key_col + j), corr_key(r, i, P.kl));
    }
  }
}

// Groups of kLanes lanes, one window each, over up to two profile sides (a
// single join).  The loop bound is warp-uniform: a warp's four groups stay
// together for the shuffles.
__global__ void __launch_bounds__(256) final_eval_kernel(EvalPair E) {
  const int lane = threadIdx.x & 31;
  const int sub = lane & (kLanes - 1);
  const int64_t total = E.side[0].ns + E.side[1].ns;
  const int64_t nwarps = static_cast<int64_t>(gridDim.x) * (blockDim.x >> 5);
  constexpr int kGroups = 32 / kLanes;
  for (int64_t g0 = ((static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x) >> 5) * kGroups;
       g0 < total; g0 += nwarps * kGroups) {
    const int64_t g = g0 + lane / kLanes;
    const bool active = g < total;
    const int s = (active && g >= E.side[0].ns) ? 1 : 0;
    const int64_t w = active ? g - (s ? E.side[0].ns : 0) : 0;
    eval_window(E.side[s], w, E.m, E.kl, sub, active);
  }
}

// The same over a batch: side k covers windows win_prefix[k] ..
// win_prefix[k + 1] - 1 of the launch.
__global__ void __launch_bounds__(256) final_eval_batch_kernel(const EvalSide* __restrict__ sides,
                                                               const int64_t* __restrict__ win_prefix,
                                                               int nsides, KeyLayout kl) {
  const int lane = threadIdx.x & 31;
  const int sub = lane & (kLanes - 1);
  const int64_t total = win_prefix[nsides];
  const int64_t nwarps = static_cast<int64_t>(gridDim.x) * (blockDim.x >> 5);
  constexpr int kGroups = 32 / kLanes;
  for (int64_t g0 = ((static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x) >> 5) * kGroups;
       g0 < total; g0 += nwarps * kGroups) {
    const int64_t g = g0 + lane / kLanes;
    const bool active = g < total;
    int lo = 0;
    if (active) {
      int hi = nsides;
      while (hi - lo > 1) {
        const int mid = (lo + hi) >> 1;
        if (win_prefix[mid] <= g) lo = mid; else hi = mid;
      }
    }
    const EvalSide& s = sides[lo];
    eval_window(s, active ? g - win_prefix[lo] : 0, s.m, kl, sub, active);
  }
}

}  // namespace scamp_gb300
