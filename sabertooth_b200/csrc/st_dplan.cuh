// Device-side planning of a batch of (profile, target) pairs for the packed
// 16-bit kernel: the same plan the host planner builds (pairs grouped by
// query, targets longest first, a tile class per query from the class rates and its critical path,
// warp tasks of 64/G targets, CTA tasks capped at one CTA's share of their
// class, CTA tasks longest first), built on the GPU so that a large batch
// needs no host pass over its pairs beyond validation.
//
// Stages (one stream, in order):
//   classify   pair -> route (empty / 16-bit / 32-bit), SoA copies for the
//              32-bit kernel, a sort key (query, target length descending)
//   sort       radix sort of the keys (stable: equal keys keep pair order)
//   estimate   per query and class: the chip's time for the query's streamed
//              cells; the batch's time with every query in its cheapest class
//   paths      the longest critical path of the queries in their cheapest classes
//   limits     for each of 32 limits on the paths: what the queries would take
//   pick       per query: the tile class under the best limit or by its own weight,
//              warp-task count, per-class totals (atomics)
//   split      per query: CTA-task count under the class's cost cap
//   order      queries sorted by class, exclusive scans of slots, warp tasks
//              and CTA tasks in that order (class segments are contiguous)
//   -- the host reads the per-class totals once, then sizes the rest --
//   emit       per query: slot records, warp tasks, CTA tasks + LPT keys
//   lpt        radix sort of CTA tasks by (class, cost descending), gather
#pragma once
#include <cstdint>

#include "../../include/sabertooth_b200.h"
#include "st_band16.cuh"
#include "st_common.cuh"
#include "st_sw16.cuh"
#include "st_tuning.h"

namespace st {

constexpr int kDpMaxClasses = 32;
constexpr uint32_t kDpNoClass = 63;  // sort key of a query with no 16-bit pairs

static_assert(kTuneLimits == 32, "a lane for each limit");
static_assert(kTuneMaxPasses <= kMaxPasses16, "a pass number has to fit the packed kernel's control word");

struct DpClass {
  uint32_t G, R, C, W;
  uint32_t team;      // a CTA's warps share each warp task's passes
  uint32_t rows;      // G * R
  uint32_t S;         // targets per warp task, 64 / G
  uint32_t max_mpad;  // the largest staged row count of the class (tune_max_rows)
  float rate;         // streamed cells per second / 1e12 (0: not considered)
};

struct DpClasses {
  DpClass c[kDpMaxClasses];
  int n;
  int table[10][8];  // forced class per (query-length bin, mean target-length bin), -1: none
  uint32_t sms;      // SMs of the device (CTA-task cap: one CTA's share on two CTAs per SM)
};

// Per-class totals, filled by pick and split with atomics, read by the host.
struct DpTotals {
  uint32_t n_query[kDpMaxClasses];
  uint32_t n_wt[kDpMaxClasses];
  uint32_t n_cta[kDpMaxClasses];
  uint32_t max_mpad[kDpMaxClasses];
  uint32_t max_cols[kDpMaxClasses];        // widest warp task
  uint32_t max_cols_multi[kDpMaxClasses];  // widest warp task of a query with several passes
  unsigned long long cost[kDpMaxClasses];  // sum of warp-task costs (the CTA-task cap)
  unsigned long long batch_ps;             // the batch's time with every query in its cheapest class
  unsigned long long longest_path, path_sum;  // of the queries in their cheapest classes, picoseconds
  uint32_t n_queries, n_wait;              // queries with 16-bit pairs, those that wait (tune_waits)
  // under each limit: cell time, longest path, scheduler rounds
  unsigned long long cells_ps[kTuneLimits], path_ps[kTuneLimits], rounds[kTuneLimits];
};

struct DpIn {
  const st_pair* pairs;
  uint32_t n;
  DeviceDb db;
  DeviceProfiles prof;
  uint32_t n_prof;
  uint32_t max_m16;  // longest query the 16-bit classes stage; longer ones take the 32-bit kernel
  uint32_t max_n16;  // longest target of a 16-bit pair
  uint32_t g16;      // gap costs inside the 16-bit kernel's range
  uint32_t tbits;    // bits of the sort key's target-length field
};

struct DpWork {
  // per pair
  uint32_t *pq, *pt;
  int32_t *pc, *pr;
  unsigned long long *keys, *keys_alt;
  uint32_t *vals, *vals_alt;  // after the sort: vals_sorted = pair ids grouped by query
  const uint32_t* vals_sorted;
  const unsigned long long* keys_sorted;
  uint32_t* list32;      // 32-bit list (static entries first, 16-bit overflows appended by the kernels)
  uint32_t* list_count;  // device count of list32
  // per query
  uint32_t *qcnt, *qstart;  // 16-bit pairs per query and their start in vals_sorted
  uint32_t *qclass, *nwt, *ncta;
  uint32_t *qkey, *qkey_alt, *qid, *qid_alt;  // queries sorted by class
  const uint32_t* qid_sorted;
  uint32_t *a_slots, *a_wt, *a_cta;  // counts in class order, then their exclusive scans
  uint32_t *o_slots, *o_wt, *o_cta;
  DpTotals* totals;
  double* est;  // per query and class: the chip's time for the query, picoseconds
};

struct DpOut {
  Sw16Slot* slots;
  Sw16WarpTask* wt;
  Sw16CtaTask* cta_raw;
  Sw16CtaTask* cta;  // LPT order, class segments in class order
  unsigned long long *cta_key, *cta_key_alt;
  uint32_t *cta_idx, *cta_idx_alt;
  const uint32_t* cta_idx_sorted;
  uint32_t n_cta;
};

__device__ __forceinline__ uint32_t dp_up4(uint32_t x) { return (x + 3u) & ~3u; }
__device__ __forceinline__ uint32_t dp_up16(uint32_t x) { return (x + 15u) & ~15u; }

__device__ __forceinline__ int dp_mbin(uint32_t m) {
  int b = 0;
  uint32_t lim = 32;
  while (b < 9 && m > lim) {
    ++b;
    lim <<= 1;
  }
  return b;
}
__device__ __forceinline__ int dp_nbin(uint32_t n) {
  int b = 0;
  uint32_t lim = 64;
  while (b < 7 && n > lim) {
    ++b;
    lim <<= 1;
  }
  return b;
}

// Shape of query m in class k.
struct DpShape {
  uint32_t P, mpad, minc, step_cost;
};
__device__ __forceinline__ DpShape dp_shape(const DpClass& k, uint32_t m) {
  DpShape s;
  s.P = (m + k.rows - 1) / k.rows;
  s.mpad = s.P * k.rows;
  s.minc = s.P > 1 ? max(32u, dp_up16(k.C * k.G)) : 32u;
  s.step_cost = k.R * k.C + 8;
  return s;
}

// Cost of a warp task whose longest target has tl residues: its wavefront steps, each of step_cost.
__device__ __forceinline__ unsigned long long dp_wt_cost(const DpClass& c, const DpShape& sh, uint32_t tl) {
  return static_cast<unsigned long long>(sh.P) * (max(sh.minc, dp_up4(tl)) / c.C) * sh.step_cost;
}

__device__ __forceinline__ unsigned long long dp_warp_sum(unsigned long long v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xFFFFFFFFu, v, o);
  return v;
}

// ---- classify: one thread per pair ----
__global__ void __launch_bounds__(256) dp_classify_kernel(const DpIn in, const DpWork w) {
  const unsigned long long sentinel = (in.tbits + 32 >= 64) ? ~0ull : ((1ull << (in.tbits + 32)) - 1);
  const uint32_t tmask = (in.tbits >= 32) ? 0xFFFFFFFFu : ((1u << in.tbits) - 1);
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < in.n; i += gridDim.x * blockDim.x) {
    const uint4 x = __ldg(reinterpret_cast<const uint4*>(in.pairs) + i);
    const uint32_t q = x.x, t = x.y;
    const int32_t radius = static_cast<int32_t>(x.w);
    w.pq[i] = q;
    w.pt[i] = t;
    w.pc[i] = static_cast<int32_t>(x.z);
    w.pr[i] = radius;
    const uint32_t m = in.prof.qlen[q];
    const uint32_t tl = in.db.length[t];
    unsigned long long key = sentinel;
    if (m != 0 && tl != 0) {
      if (radius < 0 && in.g16 && in.prof.fits8[q] && m <= in.max_m16 && tl <= in.max_n16) {
        key = (static_cast<unsigned long long>(q) << in.tbits) | (tmask - tl);
        atomicAdd(&w.qcnt[q], 1u);
      } else {
        w.list32[atomicAdd(w.list_count, 1u)] = i;
      }
    }
    w.keys[i] = key;
    w.vals[i] = i;
  }
}

// ---- 32-bit list order: longest first by the steps a warp spends on a pair ----
// passes x (streamed columns + ramp); a wide band streams one 256-row pass's window per pass, a narrow one follows
// its diagonal.  The key is inverted so that an ascending sort puts the costliest first.
__global__ void __launch_bounds__(256) dp_list_keys_kernel(const DpIn in, const DpWork w, uint32_t n_list,
                                                            unsigned long long* keys, uint32_t* vals) {
  for (uint32_t k = blockIdx.x * blockDim.x + threadIdx.x; k < n_list; k += gridDim.x * blockDim.x) {
    const uint32_t i = w.list32[k];
    const unsigned long long m = in.prof.qlen[w.pq[i]], tl = in.db.length[w.pt[i]];
    const unsigned long long P = (m + 255) / 256;
    const int32_t r = w.pr[i];
    unsigned long long cost = P * (tl + 31);
    if (r >= 0 && r <= band_ring_radius(32))
      cost = kRingLag * (m / kSw32R) + 2ull * r;
    else if (r >= 0)
      cost = P * (min(tl, 256ull + 2ull * static_cast<unsigned long long>(r)) + 31);
    cost = min(cost, (1ull << 48) - 1);
    keys[k] = ((1ull << 48) - 1) - cost;
    vals[k] = i;
  }
}

// Length of a query's j-th target, longest first, from its sort key.
struct DpLens {
  const unsigned long long* key;
  uint32_t tmask;
  __device__ __forceinline__ uint32_t operator()(uint32_t j) const {
    return tmask - (static_cast<uint32_t>(key[j]) & tmask);
  }
};
__device__ __forceinline__ DpLens dp_lens(const DpIn& in, const DpWork& w, uint32_t q) {
  return DpLens{w.keys_sorted + w.qstart[q], (in.tbits >= 32) ? 0xFFFFFFFFu : ((1u << in.tbits) - 1)};
}

// ---- estimate: one CTA per query, a warp per class ----
// Streamed cells over the rate for every class (as tuning_estimate), and the batch's total of the cheapest.
__global__ void __launch_bounds__(256) dp_estimate_kernel(const DpIn in, const DpWork w, const DpClasses cls) {
  __shared__ double s_est[kDpMaxClasses];
  const uint32_t q = blockIdx.x;
  const uint32_t np = w.qcnt[q];
  if (np == 0) return;
  const int lane = threadIdx.x & 31;
  const uint32_t m = in.prof.qlen[q];
  const DpLens tl = dp_lens(in, w, q);
  for (int k = threadIdx.x >> 5; k < cls.n; k += blockDim.x >> 5) {
    const DpClass& c = cls.c[k];
    const DpShape sh = dp_shape(c, m);
    double v = 1e300;
    if (sh.mpad <= c.max_mpad) {
      const uint32_t nw = (np + c.S - 1) / c.S;
      unsigned long long cols = 0;
      for (uint32_t x = lane; x < nw; x += 32) cols += max(sh.minc, dp_up4(tl(x * c.S)));
      cols = dp_warp_sum(cols);
      if (c.team) cols += static_cast<unsigned long long>(nw) * tune_team_cols(c.G, c.C, sh.P, c.W);
      v = static_cast<double>(cols) * c.S * sh.mpad;
      v = c.rate > 0.0f ? v / c.rate : v * 1e150;
    }
    if (lane == 0) s_est[k] = w.est[static_cast<size_t>(q) * kDpMaxClasses + k] = v;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    double best = 0.0;
    for (int k = 0; k < cls.n; ++k)
      if (s_est[k] < 1e140 && (best == 0.0 || s_est[k] < best)) best = s_est[k];
    atomicAdd(&w.totals->batch_ps, static_cast<unsigned long long>(best));
  }
}

// ---- paths, limits and pick: one warp per query, a lane per class ----
// The lane's class's cost for the query (as tuning_costs).
__device__ __forceinline__ TuneCost dp_cost(const DpIn& in, const DpWork& w, const DpClasses& cls, uint32_t q,
                                            uint32_t np, uint32_t longest) {
  const int lane = threadIdx.x & 31;
  const TuneCost none{1e300, 1e300, 1e300, 0.0};
  if (lane >= cls.n) return none;
  const double est = w.est[static_cast<size_t>(q) * kDpMaxClasses + lane];
  if (est >= 1e300) return none;
  const DpClass& c = cls.c[lane];
  const DpShape sh = dp_shape(c, in.prof.qlen[q]);
  return tune_cost(c.G, c.R, c.C, c.W, c.team != 0, sh.P, max(sh.minc, dp_up4(longest)), (np + c.S - 1) / c.S, est,
                   c.rate, static_cast<double>(w.totals->batch_ps), cls.sms);
}

// The first lane of the least v; -1 when none is below 1e300.
__device__ __forceinline__ int dp_least(double v) {
  int k = threadIdx.x & 31;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    const double ov = __shfl_xor_sync(0xFFFFFFFFu, v, o);
    const int ok = __shfl_xor_sync(0xFFFFFFFFu, k, o);
    if (ov < v || (ov == v && ok < k)) {
      v = ov;
      k = ok;
    }
  }
  return v < 1e300 ? k : -1;
}

__device__ __forceinline__ bool dp_by_limit(const DpTotals* t) {
  return tune_alike(static_cast<double>(t->longest_path), static_cast<double>(t->path_sum), t->n_queries, t->n_wait);
}

__global__ void __launch_bounds__(256) dp_path_kernel(const DpIn in, const DpWork w, const DpClasses cls) {
  const uint32_t q = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  if (q >= in.n_prof || w.qcnt[q] == 0) return;
  const TuneCost c = dp_cost(in, w, cls, q, w.qcnt[q], dp_lens(in, w, q)(0));
  const int k = dp_least(c.ps < 1e140 ? c.ps : 1e300);
  if ((threadIdx.x & 31) != max(k, 0)) return;
  atomicAdd(&w.totals->n_queries, 1u);
  if (k < 0) return;
  atomicMax(&w.totals->longest_path, static_cast<unsigned long long>(c.path) + 1);
  atomicAdd(&w.totals->path_sum, static_cast<unsigned long long>(c.path) + 1);
  if (tune_waits(c.path, static_cast<double>(w.totals->batch_ps))) atomicAdd(&w.totals->n_wait, 1u);
}

// A lane per limit here, for a batch whose paths are alike (classes forced by the table are not looked at).
__global__ void __launch_bounds__(256) dp_limit_kernel(const DpIn in, const DpWork w, const DpClasses cls) {
  const uint32_t q = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  if (q >= in.n_prof || w.qcnt[q] == 0 || !dp_by_limit(w.totals)) return;
  const int lane = threadIdx.x & 31;
  const TuneCost c = dp_cost(in, w, cls, q, w.qcnt[q], dp_lens(in, w, q)(0));
  const double limit = tune_limit(static_cast<double>(w.totals->longest_path), lane);
  TuneCost best{1e300, 1e300, 1e300, 0.0}, shortest = best;
  for (int k = 0; k < cls.n; ++k) {
    const double ps = __shfl_sync(0xFFFFFFFFu, c.ps, k);
    const TuneCost x{ps, ps, __shfl_sync(0xFFFFFFFFu, c.path, k), __shfl_sync(0xFFFFFFFFu, c.rounds, k)};
    if (x.ps >= 1e140) continue;
    if (x.path < shortest.path) shortest = x;
    if (x.path <= limit && x.ps < best.ps) best = x;
  }
  if (best.ps >= 1e140) best = shortest;
  if (best.ps >= 1e140) return;
  atomicAdd(&w.totals->cells_ps[lane], static_cast<unsigned long long>(best.ps));
  atomicMax(&w.totals->path_ps[lane], static_cast<unsigned long long>(best.path));
  atomicAdd(&w.totals->rounds[lane], static_cast<unsigned long long>(best.rounds));
}

__global__ void __launch_bounds__(256) dp_pick_kernel(const DpIn in, const DpWork w, const DpClasses cls) {
  const uint32_t q = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int lane = threadIdx.x & 31;
  if (q >= in.n_prof) return;
  const uint32_t np = w.qcnt[q];
  if (lane == 0) {
    w.qid[q] = q;
    w.qkey[q] = kDpNoClass;
    w.qclass[q] = kDpNoClass;
    w.nwt[q] = 0;
  }
  if (np == 0) return;
  const DpLens tl = dp_lens(in, w, q);
  unsigned long long sum = 0;
  for (uint32_t j = lane; j < np; j += 32) sum += tl(j);
  sum = dp_warp_sum(sum);
  const uint32_t m = in.prof.qlen[q];
  const uint32_t mean_n = static_cast<uint32_t>(sum / np);
  const double* est = w.est + static_cast<size_t>(q) * kDpMaxClasses;
  int best = -1;
  const int forced = cls.table[dp_mbin(m)][dp_nbin(mean_n)];
  if (forced >= 0 && forced < cls.n && est[forced] < 1e300) {
    best = forced;
  } else {
    const TuneCost c = dp_cost(in, w, cls, q, np, tl(0));
    const bool rated = c.est < 1e140;
    if (dp_by_limit(w.totals)) {
      const double limit =
          tune_limit(static_cast<double>(w.totals->longest_path),
                     dp_least(tune_batch_time(static_cast<double>(w.totals->cells_ps[lane]),
                                              static_cast<double>(w.totals->path_ps[lane]),
                                              static_cast<double>(w.totals->rounds[lane]), cls.sms)));
      best = dp_least(rated && c.path <= limit ? c.ps : 1e300);
      if (best < 0) best = dp_least(rated ? c.path : 1e300);
    }
    // by its own weight; or no class of the query has a rate
    if (best < 0) best = dp_least(c.est < 1e300 ? tune_weighed(c, static_cast<double>(w.totals->batch_ps)) : 1e300);
  }
  if (best < 0) return;  // cannot happen: the 16-bit route admits only queries some class stages
  const DpClass& c = cls.c[best];
  const DpShape sh = dp_shape(c, m);
  const uint32_t nw = (np + c.S - 1) / c.S;
  unsigned long long cost = 0;
  for (uint32_t x = lane; x < nw; x += 32) cost += dp_wt_cost(c, sh, tl(x * c.S));
  cost = dp_warp_sum(cost);
  if (lane == 0) {
    w.qclass[q] = static_cast<uint32_t>(best);
    w.qkey[q] = static_cast<uint32_t>(best);
    w.nwt[q] = nw;
    const uint32_t nc0 = max(sh.minc, dp_up4(tl(0)));
    atomicAdd(&w.totals->n_query[best], 1u);
    atomicAdd(&w.totals->n_wt[best], nw);
    atomicAdd(&w.totals->cost[best], cost);
    atomicMax(&w.totals->max_mpad[best], sh.mpad);
    atomicMax(&w.totals->max_cols[best], nc0);
    if (sh.P > 1) atomicMax(&w.totals->max_cols_multi[best], nc0);
  }
}

// CTA tasks of one query, by one warp: consecutive warp tasks in units of tune_cta_unit (a team class: one each), a task
// for each in a small batch (tune_cta_single); else a task ends at 128 warp tasks or at the unit nearest to where the
// query's running cost passes a multiple of the class's cap (its cost over two CTAs on every SM).
// f(t, w0, w1, cost) is called once for each task t by some lane; returns the number of tasks.
template <class F>
__device__ __forceinline__ uint32_t dp_for_each_cta(const DpClasses& cls, const DpTotals* tot, uint32_t k,
                                                    const DpShape& sh, uint32_t nw, const DpLens& tl, F&& f) {
  const DpClass& c = cls.c[k];
  const int lane = threadIdx.x & 31;
  unsigned long long wt_total = lane < cls.n ? tot->n_wt[lane] : 0u;
  wt_total = dp_warp_sum(wt_total);
  const uint32_t unit = c.team ? 1u : tune_cta_unit(wt_total, cls.sms, c.W);
  const unsigned long long cap = max(1ull, tot->cost[k] / (2ull * cls.sms));
  const bool single = c.team || tune_cta_single(wt_total, cls.sms, c.W);
  const unsigned long long half = unit * dp_wt_cost(c, sh, tl(0)) / 2;
  unsigned long long base = 0;         // cost of the warp tasks before this round's
  unsigned long long last_bucket = 0;  // of the last unit of the round before
  unsigned long long open_cost = 0;    // running cost at the start of the open task
  uint32_t n = 0, open_w = 0;          // tasks begun, first warp task of the open one
  for (uint32_t x0 = 0; x0 < nw; x0 += 32) {
    const uint32_t x = x0 + lane;
    const unsigned long long cw = x < nw ? dp_wt_cost(c, sh, tl(x * c.S)) : 0ull;
    unsigned long long incl = cw;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const unsigned long long y = __shfl_up_sync(0xFFFFFFFFu, incl, o);
      if (lane >= o) incl += y;
    }
    const unsigned long long excl = base + incl - cw;
    const unsigned long long bucket = (excl + half) / cap;
    unsigned long long before = __shfl_up_sync(0xFFFFFFFFu, bucket, unit);
    if (lane < static_cast<int>(unit)) before = last_bucket;
    const bool begin = x < nw && x % unit == 0 && (x == 0 || single || bucket != before || x % 128u == 0);
    const uint32_t mask = __ballot_sync(0xFFFFFFFFu, begin);
    const uint32_t lower = mask & ((1u << lane) - 1u);
    // the task before mine: begun by the next lower lane of the ballot, or the open one
    const int prev = lower ? 31 - __clz(lower) : 0;
    const unsigned long long pc = __shfl_sync(0xFFFFFFFFu, excl, prev);
    if (begin && x > 0)
      f(n + __popc(lower) - 1, lower ? x0 + prev : open_w, x, excl - (lower ? pc : open_cost));
    if (mask) {
      const int top = 31 - __clz(mask);
      open_w = x0 + top;
      open_cost = __shfl_sync(0xFFFFFFFFu, excl, top);
      n += __popc(mask);
    }
    base += __shfl_sync(0xFFFFFFFFu, incl, 31);
    last_bucket = __shfl_sync(0xFFFFFFFFu, bucket, 32 - unit);
  }
  if (lane == 0 && n) f(n - 1, open_w, nw, base - open_cost);
  return n;
}

// ---- split: one warp per query ----
__global__ void __launch_bounds__(256) dp_split_kernel(const DpIn in, const DpWork w, const DpClasses cls) {
  const uint32_t q = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int lane = threadIdx.x & 31;
  if (q >= in.n_prof) return;
  const uint32_t k = w.qclass[q];
  if (k == kDpNoClass) {
    if (lane == 0) w.ncta[q] = 0;
    return;
  }
  const DpShape sh = dp_shape(cls.c[k], in.prof.qlen[q]);
  const uint32_t n = dp_for_each_cta(cls, w.totals, k, sh, w.nwt[q], dp_lens(in, w, q),
                                     [](uint32_t, uint32_t, uint32_t, unsigned long long) {});
  if (lane == 0) {
    w.ncta[q] = n;
    atomicAdd(&w.totals->n_cta[k], n);
  }
}

// ---- counts in class order (one thread per position of the class-sorted queries) ----
__global__ void __launch_bounds__(256) dp_counts_kernel(const DpIn in, const DpWork w, const DpClasses cls) {
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i > in.n_prof) return;
  if (i == in.n_prof) {  // the scans run over n_prof + 1 entries: the last gives the totals
    w.a_slots[i] = 0;
    w.a_wt[i] = 0;
    w.a_cta[i] = 0;
    return;
  }
  const uint32_t q = w.qid_sorted[i];
  const uint32_t k = w.qclass[q];
  const bool has = k != kDpNoClass;
  w.a_slots[i] = has ? w.nwt[q] * cls.c[k].S : 0u;
  w.a_wt[i] = has ? w.nwt[q] : 0u;
  w.a_cta[i] = has ? w.ncta[q] : 0u;
}

// ---- emit: one warp per position of the class-sorted queries ----
__global__ void __launch_bounds__(256) dp_emit_kernel(const DpIn in, const DpWork w, const DpClasses cls,
                                                      const DpOut out) {
  const uint32_t i = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int lane = threadIdx.x & 31;
  if (i >= in.n_prof) return;
  const uint32_t q = w.qid_sorted[i];
  const uint32_t k = w.qclass[q];
  if (k == kDpNoClass) return;
  const DpClass& c = cls.c[k];
  const uint32_t np = w.qcnt[q];
  const DpShape sh = dp_shape(c, in.prof.qlen[q]);
  const uint32_t nw = w.nwt[q];
  const uint32_t* v = w.vals_sorted + w.qstart[q];
  const uint32_t o_slot = w.o_slots[i], o_wt = w.o_wt[i], o_cta = w.o_cta[i];
  for (uint32_t x = lane; x < nw; x += 32) {
    const uint32_t sb = o_slot + x * c.S;
    uint32_t ncols = sh.minc;
    for (uint32_t s = 0; s < c.S; ++s) {
      const uint32_t j = x * c.S + s;
      Sw16Slot sl{kNoPair, 0, 0, 0};
      if (j < np) {
        const uint32_t pi = v[j];
        const uint32_t t = w.pt[pi];
        const uint32_t tl = in.db.length[t];
        sl.pair = pi;
        sl.toff16 = static_cast<uint32_t>(in.db.offset[t] / 16);
        sl.tlen16 = dp_up16(tl);
        sl.tlen = tl;
        ncols = max(ncols, dp_up4(tl));
      }
      out.slots[sb + s] = sl;
    }
    out.wt[o_wt + x] = Sw16WarpTask{sb, ncols};
  }
  const unsigned long long kmask = (1ull << 44) - 1;
  dp_for_each_cta(cls, w.totals, k, sh, nw, dp_lens(in, w, q),
                  [&](uint32_t j, uint32_t w0, uint32_t w1, unsigned long long cost) {
                    const uint32_t t = o_cta + j;
                    out.cta_raw[t] = Sw16CtaTask{q, o_wt + w0, o_wt + w1, sh.mpad};
                    out.cta_key[t] = (static_cast<unsigned long long>(k) << 44) | (kmask - min(cost, kmask));
                    out.cta_idx[t] = t;
                  });
}

__global__ void __launch_bounds__(256) dp_gather_cta_kernel(const DpOut out) {
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < out.n_cta) out.cta[i] = out.cta_raw[out.cta_idx_sorted[i]];
}

__global__ void __launch_bounds__(256) dp_iota_kernel(uint32_t* v, uint32_t n) {
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) v[i] = i;
}

}  // namespace st
