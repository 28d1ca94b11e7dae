// Prefilter evidence, chaining and gate on the device: the reference's
// segment-evidence stage (xdrop = 0) of prefilter_query, src/prefilter.rs:
//   evaluate_block_kadane  :1412-1493  group hits by target, keep the
//                                      max_diagonals diagonals with the most hits
//                                      (top_diagonals :1194-1225), one job per
//                                      diagonal with its window
//   score_and_gate         :1498-1660  best ungapped segment per job, best single
//                                      segment or chain of two co-linear
//                                      segments, gate, region
//   ranking                :1074-1083  score descending, target ascending,
//                                      max_candidates per query
// for many queries at once.  Pipeline (one stream, no host round trip):
//   keys     one thread per hit: key = (query, target, diagonal + max_m) with the
//            query position below it; hits outside the query or the target get the
//            key of a query id past the last profile (they sort last and are skipped)
//   sort     radix sort of the keys by (query, target, diagonal) (CUB).  The
//            position travels in the key's low bits, which are not sorted: 8
//            bytes a hit and pass where a value beside the key makes it 12.
//            Only where the four fields need more than 64 bits are the
//            positions sorted as values.  8 M hits of 400 queries: the whole
//            path 1.67 -> 1.55 ms.
//   groups   start of each (query, target) run of the sorted keys (CUB select)
//   count    one thread per group: min_hits / diag_hits tests and the number of
//            jobs, min(distinct diagonals, max_diagonals, 16)
//   scan     job offsets (CUB exclusive sum)
//   emit     one thread per group: the top diagonals by hit count (stable on the
//            ascending diagonal order) and their windows, written as jobs
//   score    one job per lane with refill, jobs of one query share its profile
//            staged in shared memory: kadane_score over the window
//   screen   groups that may pass (several diagonals, or one at the gate) to a
//            work list
//   chain    one thread per listed group: best segment, best chain, gate,
//            region, candidate slot + flag; kadane_segment positions only for
//            the jobs a chain test or a region may read (the reference's pos_of)
//   compact  candidates in (query, target) order (CUB select)
//   rank     stable radix sort by (query, 2^31 - 1 - score) keeps target order
//            inside equal scores; per-query cut to max_candidates; gather
#pragma once
#include "st_common.cuh"
#include "st_ungapped.cuh"

namespace st {

constexpr int kGateMaxDiags = 16;  // jobs per target (src/prefilter.rs:1459, top.iter().take(16))

struct GateCandidate {  // the layout of st_candidate
  uint32_t query;
  uint32_t target;
  uint32_t hits;
  int32_t diag_score;
  int64_t best_diag;
  uint32_t t_lo;
  uint32_t t_hi;
};
static_assert(sizeof(GateCandidate) == 32, "candidate layout");

struct GateJob {
  uint32_t query;
  uint32_t target;
  int32_t diag;
  uint32_t lo;
  uint32_t hi;
};

struct GateSeedHit {  // the layout of st_seed_hit
  uint32_t query;
  uint32_t target;
  int32_t diag;
  uint32_t qpos;
};

// Counters, the layout of st_prefilter_stats.
struct GateStats {
  unsigned long long targets_hit;
  unsigned long long targets_evaluated;
  unsigned long long diagonals_scored;
  unsigned long long chains_used;
  unsigned long long candidates;
  unsigned long long candidates_capped;
  unsigned long long hits_rejected;
};

struct GateConf {
  uint32_t min_hits;
  uint32_t diag_hits;
  uint32_t kmax;  // min(max_diagonals, 16)
  uint32_t window;
  uint32_t span;
  int32_t min_score;
  int32_t open;
  int32_t ext;
  uint32_t max_cand;  // 0 = all
  uint32_t regions;
  // key layout: (query << (tbits + dbits) | target << dbits | (diag + doff)) << pbits, and the query position in the
  // low pbits
  uint32_t pbits;  // 0: the positions are sorted beside the keys
  uint32_t tbits;
  uint32_t dbits;
  uint32_t doff;
  uint32_t n_prof;  // query ids are < n_prof; n_prof marks rejected hits
  uint32_t stride;  // staged profile row stride: >= every hit query's length rounded to 16, + 32
};

__device__ __forceinline__ uint32_t gate_key_query(uint64_t k, const GateConf& g) {
  return static_cast<uint32_t>(k >> (g.tbits + g.dbits + g.pbits));
}
__device__ __forceinline__ uint32_t gate_key_target(uint64_t k, const GateConf& g) {
  return static_cast<uint32_t>((k >> (g.dbits + g.pbits)) & ((1ull << g.tbits) - 1));
}
__device__ __forceinline__ int32_t gate_key_diag(uint64_t k, const GateConf& g) {
  return static_cast<int32_t>(static_cast<int64_t>((k >> g.pbits) & ((1ull << g.dbits) - 1)) - g.doff);
}

__device__ __forceinline__ uint64_t gate_key(uint32_t query, uint32_t target, int32_t diag, uint32_t qpos,
                                             const GateConf& g) {
  const uint64_t k = (static_cast<uint64_t>(query) << (g.tbits + g.dbits)) | (static_cast<uint64_t>(target) << g.dbits) |
                     static_cast<uint64_t>(static_cast<int64_t>(diag) + g.doff);
  return g.pbits ? (k << g.pbits) | qpos : k;
}

// Adds each thread's count to a counter; called by every thread of the block
// once, after its loop (all 32 lanes of each warp present).
__device__ __forceinline__ void gate_flush(unsigned long long* ctr, unsigned long long v) {
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xFFFFFFFFu, v, o);
  if ((threadIdx.x & 31) == 0 && v) atomicAdd(ctr, v);
}

// The same with one atomic a block, for short even loops whose every warp has a
// count: a counter is a single address, which takes about one atomic a
// nanosecond (seed_post_count_kernel of 38,000 warps 187 -> 128 us).  Kernels of
// uneven warps keep the form above: the barrier holds their early warps' places
// (gate_count_kernel 108 -> 147 us with this one).
__device__ __forceinline__ void gate_flush_block(unsigned long long* ctr, unsigned long long v) {
  __shared__ unsigned long long s_sum;
  if (threadIdx.x == 0) s_sum = 0;
  __syncthreads();
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xFFFFFFFFu, v, o);
  if ((threadIdx.x & 31) == 0 && v) atomicAdd(&s_sum, v);
  __syncthreads();
  if (threadIdx.x == 0 && s_sum) atomicAdd(ctr, s_sum);
  __syncthreads();  // before the next counter of the block
}

__global__ void __launch_bounds__(256) gate_keys_kernel(const GateSeedHit* hits, uint64_t n, DeviceDb db,
                                                        const uint32_t* qlen, GateConf g, uint64_t* keys,
                                                        uint32_t* vals, GateStats* st) {
  const uint64_t bad = static_cast<uint64_t>(g.n_prof) << (g.tbits + g.dbits + g.pbits);
  unsigned long long rejected = 0;
  for (uint64_t i = static_cast<uint64_t>(blockIdx.x) * blockDim.x + threadIdx.x; i < n;
       i += static_cast<uint64_t>(gridDim.x) * blockDim.x) {
    const GateSeedHit h = hits[i];
    bool ok = h.query < g.n_prof && h.target < db.n_seqs;
    if (ok) {
      const int64_t tpos = static_cast<int64_t>(h.qpos) + h.diag;
      ok = h.qpos < qlen[h.query] && tpos >= 0 && tpos < static_cast<int64_t>(db.length[h.target]);
    }
    keys[i] = ok ? gate_key(h.query, h.target, h.diag, h.qpos, g) : bad;
    if (!g.pbits) vals[i] = h.qpos;
    rejected += ok ? 0 : 1;
  }
  gate_flush(&st->hits_rejected, rejected);
}

// Flag of the first hit of each (query, target) run in the sorted keys.
struct GateHeadFlag {
  const uint64_t* keys;
  uint32_t shift;  // dbits + pbits
  __host__ __device__ bool operator()(uint32_t i) const {
    return i == 0 || (keys[i] >> shift) != (keys[i - 1] >> shift);
  }
};

struct GateGroups {
  const uint64_t* keys;  // sorted
  const uint32_t* vals;  // query positions, in key order, where the keys do not hold them
  const uint32_t* start; // first hit of each group
  const uint32_t* n_groups;
  uint32_t n_hits;
};

__device__ __forceinline__ void gate_group_range(const GateGroups& G, uint32_t gi, uint32_t ng, uint32_t& s,
                                                 uint32_t& e) {
  s = G.start[gi];
  e = gi + 1 < ng ? G.start[gi + 1] : G.n_hits;
}

// Query position of the sorted hit i with key k.
__device__ __forceinline__ uint32_t gate_pos(const GateGroups& G, uint32_t i, uint64_t k, const GateConf& g) {
  return g.pbits ? static_cast<uint32_t>(k & ((1ull << g.pbits) - 1)) : G.vals[i];
}

// ns[g] = jobs of group g (0 when the target is dropped); entries from the last
// group to n_hits are zeroed so the exclusive sum over n_hits + 1 entries ends
// at the total job count.
__global__ void __launch_bounds__(256) gate_count_kernel(GateGroups G, GateConf g, uint32_t* ns, GateStats* st) {
  const uint32_t ng = *G.n_groups;
  unsigned long long n_hit = 0, n_eval = 0;
  for (uint32_t gi = blockIdx.x * blockDim.x + threadIdx.x; gi <= G.n_hits; gi += gridDim.x * blockDim.x) {
    uint32_t jobs = 0, evaluated = 0, hit = 0;
    if (gi < ng) {
      uint32_t s, e;
      gate_group_range(G, gi, ng, s, e);
      const uint64_t k0 = G.keys[s];
      if (gate_key_query(k0, g) < g.n_prof) {
        hit = 1;
        if (e - s >= g.min_hits) {
          uint32_t runs = 0, best = 0, cnt = 0;
          uint64_t prev = ~0ull;
          for (uint32_t i = s; i < e; ++i) {
            const uint64_t k = G.keys[i] >> g.pbits;
            if (k != prev) {
              ++runs;
              cnt = 0;
              prev = k;
            }
            ++cnt;
            best = max(best, cnt);
          }
          if (best >= g.diag_hits) {
            jobs = min(runs, g.kmax);
            evaluated = 1;
          }
        }
      }
    }
    ns[gi] = jobs;
    n_hit += hit;
    n_eval += evaluated;
  }
  gate_flush(&st->targets_hit, n_hit);
  gate_flush(&st->targets_evaluated, n_eval);
}

struct GateRun {
  int32_t diag;
  uint32_t count;
  uint32_t qmin;
  uint32_t qmax;
};

// Jobs of each kept group: its KMAX best diagonals by hit count (a run goes
// before the first kept run with a smaller count, so equal counts keep the
// ascending diagonal order), with windows (src/prefilter.rs:1459-1474).
template <int KMAX>
__global__ void __launch_bounds__(128) gate_emit_kernel(GateGroups G, GateConf g, DeviceDb db, const uint32_t* qlen,
                                                        const uint32_t* ns, const uint32_t* joff, GateJob* jobs) {
  const uint32_t ng = *G.n_groups;
  for (uint32_t gi = blockIdx.x * blockDim.x + threadIdx.x; gi < ng; gi += gridDim.x * blockDim.x) {
    if (ns[gi] == 0) continue;
    uint32_t s, e;
    gate_group_range(G, gi, ng, s, e);
    GateRun top[KMAX];
    uint32_t nt = 0;
    uint32_t i = s;
    while (i < e) {
      const uint64_t k = G.keys[i];
      const uint32_t p0 = gate_pos(G, i, k, g);
      GateRun r{gate_key_diag(k, g), 0, p0, p0};
      uint32_t j = i + 1;
      for (; j < e; ++j) {
        const uint64_t kj = G.keys[j];
        if (kj >> g.pbits != k >> g.pbits) break;
        const uint32_t p = gate_pos(G, j, kj, g);
        r.qmin = min(r.qmin, p);
        r.qmax = max(r.qmax, p);
      }
      r.count = j - i;
      i = j;
      // pos = kept runs with count >= r.count
      uint32_t pos = 0;
#pragma unroll
      for (int t = 0; t < KMAX; ++t) pos += (static_cast<uint32_t>(t) < nt && top[t].count >= r.count) ? 1u : 0u;
      if (pos < g.kmax) {
#pragma unroll
        for (int t = KMAX - 1; t > 0; --t)
          if (static_cast<uint32_t>(t) > pos) top[t] = top[t - 1];
#pragma unroll
        for (int t = 0; t < KMAX; ++t)
          if (static_cast<uint32_t>(t) == pos) top[t] = r;
        nt = min(nt + 1, g.kmax);
      }
    }
    const uint64_t k0 = G.keys[s];
    const uint32_t q = gate_key_query(k0, g), t = gate_key_target(k0, g);
    const int64_t m = qlen[q], n = db.length[t];
    GateJob* out = jobs + joff[gi];
#pragma unroll
    for (int k = 0; k < KMAX; ++k) {
      if (static_cast<uint32_t>(k) >= nt) break;
      const int32_t d = top[k].diag;
      // diag_range (src/ungapped.rs:38-46), then the window around the hits
      int64_t lo = i64max(-static_cast<int64_t>(d), 0), hi = i64min(m, n - d);
      if (hi <= lo) lo = hi = 0;
      if (g.window > 0) {
        const int64_t a = top[k].qmin > g.window ? static_cast<int64_t>(top[k].qmin - g.window) : 0;
        const int64_t b = static_cast<int64_t>(top[k].qmax) + g.span + g.window;
        lo = i64max(lo, a);
        hi = i64min(hi, b);
      }
      hi = i64max(hi, lo);
      out[k] = GateJob{q, t, d, static_cast<uint32_t>(lo), static_cast<uint32_t>(hi)};
    }
  }
}

struct GateSegParams {
  DeviceDb db;
  DeviceProfiles prof;
  const GateJob* jobs;
  const uint32_t* n_groups;
  const uint32_t* joff;  // total jobs at joff[n_groups]
  int32_t* score;
  uint32_t max_m_pad;
  uint32_t chunk;  // jobs per CTA
};

// kadane_score (src/ungapped.rs:53-62) of each job over its window: a CTA takes a chunk of jobs and scores each run of
// one query inside it with diag_score_run.
__global__ void __launch_bounds__(256) gate_score_kernel(const GateSegParams prm) {
  extern __shared__ __align__(16) int8_t smem[];
  __shared__ uint32_t s_run_end, s_next;
  const uint32_t n = prm.joff[*prm.n_groups];
  const uint32_t stride = prm.max_m_pad;
  const uint64_t c0 = static_cast<uint64_t>(blockIdx.x) * prm.chunk;
  if (c0 >= n) return;
  const uint32_t nc = min(n - static_cast<uint32_t>(c0), prm.chunk);
  const GateJob* chunk = prm.jobs + c0;
  uint32_t a = 0;
  while (a < nc) {
    const uint32_t q = chunk[a].query;
    if (threadIdx.x < 32) {
      uint32_t e = a;
      for (;;) {
        const uint32_t k = e + threadIdx.x;
        const uint32_t ball = __ballot_sync(0xFFFFFFFFu, k < nc && chunk[k].query == q);
        if (ball != 0xFFFFFFFFu) {
          e += __ffs(~ball) - 1;
          break;
        }
        e += 32;
      }
      if (threadIdx.x == 0) {
        s_run_end = e;
        s_next = blockDim.x;
      }
    }
    diag_stage(prm.prof, q, stride, smem);
    __syncthreads();
    const uint32_t b = s_run_end;
    const GateJob* run = chunk + a;
    diag_score_run<true>(
        smem + 16, stride, prm.prof.fits8[q] != 0, prm.prof.p32[q], static_cast<int32_t>(prm.prof.stride32[q]),
        static_cast<int32_t>(prm.prof.qlen[q]) - 1, b - a, &s_next, prm.score + c0 + a, [&](uint32_t j) {
          const GateJob jb = run[j];
          return DiagWindow{prm.db.arena + prm.db.offset[jb.target], jb.diag, static_cast<int32_t>(jb.lo) + jb.diag,
                            static_cast<int32_t>(jb.hi) + jb.diag};
        });
    a = b;
  }
}

// kadane_segment (src/ungapped.rs:69-88) of one job from the profile in global
// memory: best score, start of the run that first reaches it and its end
// (0, 0 when the best is 0).  Used only for the jobs whose positions decide a
// chain or a region.  Target residues come as 16-byte vectors and the 16
// profile loads of a vector are independent of each other; cells outside the
// window score 0, which moves neither the best nor where it is first reached.
__device__ int32_t gate_kadane_segment(const DeviceProfiles& prof, const DeviceDb& db, const GateJob& jb, int32_t& qs,
                                       int32_t& qe) {
  int32_t best = 0, cur = 0, bs = 0, be = 0, cs = 0;
  if (jb.hi > jb.lo) {
    const uint8_t* t = db.arena + db.offset[jb.target];
    const bool narrow = prof.fits8[jb.query] != 0;
    const int8_t* p8 = prof.p8[jb.query];
    const int32_t* p32 = prof.p32[jb.query];
    const int32_t s8 = static_cast<int32_t>(prof.stride8[jb.query]), s32 = static_cast<int32_t>(prof.stride32[jb.query]);
    const int32_t d = jb.diag, lo = static_cast<int32_t>(jb.lo), hi = static_cast<int32_t>(jb.hi);
    const int32_t p0 = lo + d, p1 = hi + d;
    for (int32_t pa = p0 & ~15; pa < p1; pa += 16) {
      const uint4 v = *reinterpret_cast<const uint4*>(t + pa);
      const uint32_t w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
      for (int bb = 0; bb < 16; ++bb) {
        const uint32_t r = (w[bb >> 2] >> ((bb & 3) * 8)) & 0xFFu;
        const int32_t q = pa + bb - d;
        const bool in = q >= lo && q < hi;
        const int32_t qc = min(max(q, lo), hi - 1);
        const int32_t sv = narrow ? static_cast<int32_t>(p8[static_cast<int32_t>(r) * s8 + qc])
                                  : p32[static_cast<int32_t>(r) * s32 + qc];
        const int32_t s = in ? sv : 0;
        if (cur <= 0) {
          cur = s;
          cs = q;
        } else {
          cur = wadd(cur, s);
        }
        if (cur > best) {
          best = cur;
          bs = cs;
          be = q;
        }
      }
    }
  }
  qs = bs;
  qe = be;
  return best;
}

__device__ __forceinline__ int32_t gate_gap_cost(int32_t open, int32_t ext, uint32_t len) {
  return len == 0 ? 0 : wadd(open, static_cast<int32_t>((len - 1u) * static_cast<uint32_t>(ext)));
}

// Groups that may pass the gate: every group with more than one diagonal or
// with its one diagonal at or above the gate goes to a work list (the order of
// the list does not matter: each group writes its own slot).  Groups left out
// keep the zero flag written before.  A CTA takes the places of its tile of
// groups with one atomic: one a warp on the one counter was 280 us for 14 M
// windows' groups.
constexpr uint32_t kScreenTile = 2048;
__global__ void __launch_bounds__(256) gate_screen_kernel(GateGroups G, GateConf g, const uint32_t* joff,
                                                          const int32_t* score, uint32_t* work, uint32_t* n_work) {
  constexpr uint32_t kPer = kScreenTile / 256;
  __shared__ uint32_t s_warp[8], s_base;
  const uint32_t ng = *G.n_groups;
  const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  for (uint32_t t0 = blockIdx.x * kScreenTile; t0 < ng; t0 += gridDim.x * kScreenTile) {
    uint32_t bits = 0;  // this thread's groups t0 + 256 i + threadIdx.x that may pass
#pragma unroll
    for (uint32_t i = 0; i < kPer; ++i) {
      const uint32_t gi = t0 + 256 * i + threadIdx.x;
      if (gi < ng) {
        const uint32_t j0 = joff[gi], nsg = joff[gi + 1] - j0;
        if (nsg > 1 || (nsg == 1 && score[j0] >= g.min_score)) bits |= 1u << i;
      }
    }
    const uint32_t cnt = __popc(bits);
    uint32_t incl = cnt;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t y = __shfl_up_sync(0xFFFFFFFFu, incl, o);
      if (lane >= o) incl += y;
    }
    if (lane == 31) s_warp[warp] = incl;
    __syncthreads();
    if (threadIdx.x == 0) {
      uint32_t sum = 0;
      for (int w = 0; w < 8; ++w) {
        const uint32_t x = s_warp[w];
        s_warp[w] = sum;
        sum += x;
      }
      s_base = sum ? atomicAdd(n_work, sum) : 0u;
    }
    __syncthreads();
    uint32_t at = s_base + s_warp[warp] + incl - cnt;
    for (uint32_t b = bits; b; b &= b - 1) work[at++] = t0 + 256 * (__ffs(b) - 1) + threadIdx.x;
    __syncthreads();
  }
}

// Best single segment (first maximum in job order) or best chain x -> y of two
// co-linear segments (first maximum in (x, y) order), the gate and the region
// (src/prefilter.rs:1577-1657, region :1269-1278), one thread per listed group.
// Segment positions decide only the pairs whose chain would beat the best single
// segment, and the region: each thread marks the jobs it needs, the CTA packs
// them and walks them one a thread, so that a warp walks 32 windows where the
// threads' own few left most of its lanes waiting, and the scores and diagonals
// of a group are read at once (14 M windows of 150 queries: 545 -> 275 us).
template <int KMAX>
constexpr int kChainThreads = KMAX <= 4 ? 256 : 128;  // 12 or 24 KB of shared memory a CTA
template <int KMAX>
__global__ void __launch_bounds__(kChainThreads<KMAX>) gate_chain_kernel(
    GateGroups G, GateConf g, DeviceDb db, DeviceProfiles prof, const uint32_t* joff, const GateJob* jobs,
    const int32_t* score, const uint32_t* work, const uint32_t* n_work, GateCandidate* cand, uint8_t* flag,
    GateStats* st) {
  constexpr uint32_t T = kChainThreads<KMAX>;
  __shared__ uint32_t s_job[T * KMAX], s_warp[T / 32];
  __shared__ int2 s_pos[T * KMAX];  // query positions of the first and last cell of the job's best segment
  const uint32_t ng = *G.n_groups;
  const uint32_t nw = *n_work;
  const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  unsigned long long n_chained = 0;
  for (uint32_t w0 = blockIdx.x * T; w0 < nw; w0 += gridDim.x * T) {
    const bool on = w0 + threadIdx.x < nw;
    uint32_t gi = 0, j0 = 0, nsg = 0, bi = 0, need = 0;
    int32_t best = 0;
    int32_t seg[KMAX], dg[KMAX];  // the group's segment scores (0 past its last) and diagonals
#pragma unroll
    for (int k = 0; k < KMAX; ++k) seg[k] = dg[k] = 0;
    // pair(x, y, c, dx, dy) for the ordered pairs whose chain score beats the best single segment
    auto pairs = [&](auto&& pair) {
#pragma unroll(KMAX <= 4 ? KMAX : 1)
      for (uint32_t x = 0; x < KMAX; ++x) {
        const int32_t sx = seg[x], dx = dg[x];
        if (sx <= 0) continue;
#pragma unroll(KMAX <= 4 ? KMAX : 1)
        for (uint32_t y = 0; y < KMAX; ++y) {
          if (x == y) continue;
          const int32_t sy = seg[y], dy = dg[y];
          if (sy <= 0 || dx == dy) continue;
          const uint32_t len = static_cast<uint32_t>(dy > dx ? dy - dx : dx - dy);
          const int32_t c = wsub(wadd(sx, sy), gate_gap_cost(g.open, g.ext, len));
          if (c > best) pair(x, y, c, dx, dy);
        }
      }
    };
    if (on) {
      gi = work[w0 + threadIdx.x];
      j0 = joff[gi];
      nsg = joff[gi + 1] - j0;
#pragma unroll
      for (uint32_t k = 0; k < KMAX; ++k)
        if (k < nsg) {
          seg[k] = score[j0 + k];
          dg[k] = jobs[j0 + k].diag;
        }
#pragma unroll
      for (uint32_t k = 0; k < KMAX; ++k)
        if (seg[k] > best) {
          best = seg[k];
          bi = k;
        }
      if (nsg > 1) pairs([&](uint32_t x, uint32_t y, int32_t, int32_t, int32_t) { need |= 1u << x | 1u << y; });
      if (g.regions && best >= g.min_score) need |= 1u << bi;
    }
    const uint32_t cnt = __popc(need);
    uint32_t incl = cnt;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t v = __shfl_up_sync(0xFFFFFFFFu, incl, o);
      if (lane >= o) incl += v;
    }
    if (lane == 31) s_warp[warp] = incl;
    __syncthreads();
    uint32_t base = incl - cnt, total = 0;
#pragma unroll
    for (uint32_t v = 0; v < T / 32; ++v) {
      base += v < warp ? s_warp[v] : 0u;
      total += s_warp[v];
    }
    {
      uint32_t at = base;
      for (uint32_t m = need; m; m &= m - 1) s_job[at++] = j0 + (__ffs(m) - 1);
    }
    __syncthreads();
    for (uint32_t i = threadIdx.x; i < total; i += T) {
      int32_t a, b;
      gate_kadane_segment(prof, db, jobs[s_job[i]], a, b);
      s_pos[i] = make_int2(a, b);
    }
    __syncthreads();
    auto pos = [&](uint32_t x) { return s_pos[base + __popc(need & ((1u << x) - 1u))]; };
    if (on) {
      int32_t chain = INT32_MIN;
      uint32_t cx = 0, cy = 0;
      if (need && nsg > 1)
        pairs([&](uint32_t x, uint32_t y, int32_t c, int32_t dx, int32_t dy) {
          if (c <= chain) return;
          const int32_t qex = pos(x).y, qsy = pos(y).x;
          if (qex < qsy && static_cast<int64_t>(qex) + dx < static_cast<int64_t>(qsy) + dy) {
            chain = c;
            cx = x;
            cy = y;
          }
        });
      int32_t sum;
      uint32_t u0, u1;
      if (chain > best) {
        ++n_chained;
        sum = chain;
        u0 = cx;
        u1 = cy;
      } else {
        sum = best;
        u0 = u1 = bi;
      }
      if (sum >= g.min_score) {
        uint32_t s, e;
        gate_group_range(G, gi, ng, s, e);
        uint32_t rlo = 0, rhi = 0xFFFFFFFFu;
        if (g.regions) {
          const int2 p0 = pos(u0), p1 = pos(u1);
          const int64_t d0 = jobs[j0 + u0].diag, d1 = jobs[j0 + u1].diag;
          const int64_t a0 = i64max(p0.x + d0, 0), b0 = i64max(p0.y + d0, 0);
          const int64_t a1 = i64max(p1.x + d1, 0), b1 = i64max(p1.y + d1, 0);
          rlo = static_cast<uint32_t>(i64min(a0, a1));
          rhi = static_cast<uint32_t>(i64max(b0, b1));
        }
        const GateJob jb = jobs[j0];
        cand[gi] = GateCandidate{jb.query, jb.target, e - s, sum, static_cast<int64_t>(jobs[j0 + bi].diag), rlo, rhi};
        flag[gi] = 1;
      }
    }
    __syncthreads();  // the shared lists are written again in the next round
  }
  gate_flush(&st->chains_used, n_chained);
}

// Rank keys of the kept candidates (sel: their group slots, in (query, target)
// order): (query, 2^31 - 1 - score) and the slot.
__global__ void __launch_bounds__(256) gate_rank_keys_kernel(const GateCandidate* cand, const uint32_t* sel,
                                                             const uint32_t* n_cand, uint64_t* keys, uint32_t* idx) {
  const uint32_t n = *n_cand;
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    const uint32_t j = sel[i];
    const GateCandidate c = cand[j];
    keys[i] = (static_cast<uint64_t>(c.query) << 31) | static_cast<uint64_t>(0x7FFFFFFF - c.diag_score);
    idx[i] = j;
  }
}

// First and last rank position of every query in the ranked list.
__global__ void __launch_bounds__(256) gate_query_bounds_kernel(const uint64_t* keys, const uint32_t* n_cand,
                                                                uint32_t* qfirst, uint32_t* qcount) {
  const uint32_t n = *n_cand;
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    const uint32_t q = static_cast<uint32_t>(keys[i] >> 31);
    if (i == 0 || static_cast<uint32_t>(keys[i - 1] >> 31) != q) qfirst[q] = i;
    if (i + 1 == n || static_cast<uint32_t>(keys[i + 1] >> 31) != q) qcount[q] = i + 1;  // end, made a count below
  }
}

// kept[q] = min(count, max_cand) for every query id (qcount holds the end).
__global__ void __launch_bounds__(256) gate_query_kept_kernel(const uint32_t* qfirst, const uint32_t* qend,
                                                              uint32_t n_prof, uint32_t max_cand, uint32_t* kept) {
  for (uint32_t q = blockIdx.x * blockDim.x + threadIdx.x; q <= n_prof; q += gridDim.x * blockDim.x) {
    uint32_t c = 0;
    if (q < n_prof) {
      c = qend[q] - qfirst[q];
      if (max_cand && c > max_cand) c = max_cand;
    }
    kept[q] = c;
  }
}

// out[pos] = the candidate of rank position i, pos = i without a cap, else the
// query's output offset + its rank inside the query (rank < max_cand).
__global__ void __launch_bounds__(256) gate_gather_kernel(const GateCandidate* cand, const uint64_t* keys,
                                                          const uint32_t* idx, const uint32_t* n_cand,
                                                          uint32_t max_cand, const uint32_t* qfirst,
                                                          const uint32_t* koff, GateCandidate* out) {
  const uint32_t n = *n_cand;
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    if (max_cand == 0) {
      out[i] = cand[idx[i]];
    } else {
      const uint32_t q = static_cast<uint32_t>(keys[i] >> 31);
      const uint32_t r = i - qfirst[q];
      if (r < max_cand) out[koff[q] + r] = cand[idx[i]];
    }
  }
}

// Final counters: diagonals scored, candidates kept and cut.
__global__ void gate_finish_kernel(const uint32_t* n_groups, const uint32_t* joff, const uint32_t* n_cand,
                                   const uint32_t* koff, uint32_t n_prof, uint32_t max_cand, GateStats* st,
                                   unsigned long long* n_out) {
  const uint32_t nj = joff[*n_groups];
  const uint32_t nc = *n_cand;
  const uint32_t kept = max_cand ? koff[n_prof] : nc;
  st->diagonals_scored += nj;
  st->candidates += kept;
  st->candidates_capped += nc - kept;
  *n_out = kept;
}

}  // namespace st
