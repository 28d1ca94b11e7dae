// Seed hits on the device: the seed stage of the reference's prefilter_query
// (src/prefilter.rs:816-995) over a device-resident seed index.
//
// Index (SeedIndex, src/index.rs:1059-1074 window_ok): every window of every
// database sequence whose care positions (the seed pattern's '1's) hold codes
// < 20, keyed by code = care residues in base 20; a direct table of 20^w + 1
// offsets (w <= 7) over (sequence, window start) postings, filled by one warp
// per sequence with one atomic counter per code (the order inside a code does
// not matter: hits are grouped by a sort later).
//
// Queries, one warp per window (query, start):
//   count  eligibility (no care residue >= 20 for sequence queries), the number
//          of k-mers over the 20 standard residues scoring >= kmer_score from a
//          histogram of partial sums pruned at the threshold (the counting pass
//          of cap_boundary, :571-609), and, above the cap, the boundary score t*
//          and how many ties at t* are kept;
//   emit   the window's k-mers by a depth-first walk in rank-lexicographic order
//          with exact suffix-maximum pruning (top_kmers, :470-568): every k-mer
//          above t* (or >= the threshold when not capped) and the first ties at
//          t* in that order — the first `cap` k-mers of the canonical order;
//          the query's own k-mer is added when it is not among them (exact seeds);
//   posts  each k-mer's posting count (skipped above max_seed_occ, push_seed
//          :853-869), then one hit (query, target, tpos - qpos, qpos) per posting.
#pragma once
#include "st_common.cuh"
#include "st_gate.cuh"

namespace st {

constexpr int kSeedMaxW = 7;        // direct table: 20^7 + 1 offsets
constexpr int kSeedAA = 20;         // standard residues
constexpr int kSeedMaxBins = 1024;  // partial-sum histogram width (score range of a window above the threshold)
constexpr uint32_t kSeedNone = 0xFFFFFFFFu;

struct SeedPat {
  uint32_t w;
  uint32_t span;
  uint32_t offs[12];
};

struct SeedPost {
  uint32_t target;
  uint32_t tpos;
};

// A query position's 20 standard residues by score descending, residue
// ascending (sorted_row, src/prefilter.rs:433-441).
struct SeedRow {
  int32_t sc[kSeedAA];
  uint8_t res[kSeedAA];
};

struct SeedWin {  // per window: boundary of the kept set
  int32_t tstar;  // INT32_MIN: not capped
  uint32_t need;  // ties at t* kept
};

struct SeedSeed {
  uint32_t code;  // kSeedNone: an unused exact-seed slot
  uint32_t window;
};

struct SeedStatsDev {  // the layout of st_seed_stats
  unsigned long long windows, windows_skipped, kmers_generated, windows_at_cap, exact_seeds_added, seeds,
      postings_visited, seeds_over_occ_cap, postings_skipped_occ, errors;
};

__device__ __forceinline__ bool seed_window_code(const uint8_t* s, const SeedPat& p, uint32_t& code) {
  uint32_t c = 0;
  for (uint32_t i = 0; i < p.w; ++i) {
    const uint32_t r = s[p.offs[i]];
    if (r >= kSeedAA) return false;
    c = c * kSeedAA + r;
  }
  code = c;
  return true;
}

// One warp per sequence, lanes over its window starts.
template <bool FILL>
__global__ void __launch_bounds__(256) seed_index_kernel(DeviceDb db, SeedPat p, uint32_t* cnt, SeedPost* post) {
  const uint32_t lane = threadIdx.x & 31;
  const uint32_t warps = gridDim.x * (blockDim.x / 32);
  for (uint32_t s = blockIdx.x * (blockDim.x / 32) + threadIdx.x / 32; s < db.n_seqs; s += warps) {
    const uint32_t n = db.length[s];
    if (n < p.span) continue;
    const uint8_t* t = db.arena + db.offset[s];
    for (uint32_t st = lane; st + p.span <= n; st += 32) {
      uint32_t code;
      if (!seed_window_code(t + st, p, code)) continue;
      if (FILL)
        post[atomicAdd(&cnt[code], 1u)] = SeedPost{s, st};
      else
        atomicAdd(&cnt[code], 1u);
    }
  }
}

// One warp per query row: a residue's place is the number of residues before it (higher score, or the same and a
// smaller code), counted over the lanes.  (One thread per row with an insertion sort: 26 us for one query, the
// dependent swaps of 20 entries in local memory.)
__global__ void __launch_bounds__(128) seed_sort_rows_kernel(DeviceProfiles prof, const uint32_t* qids,
                                                             const uint32_t* row0, SeedRow* rows) {
  const uint32_t qi = blockIdx.x;
  const uint32_t q = qids[qi];
  const uint32_t m = prof.qlen[q];
  const int32_t* p32 = prof.p32[q];
  const uint32_t s32 = prof.stride32[q];
  const uint32_t lane = threadIdx.x & 31;
  const uint32_t warps = gridDim.y * (blockDim.x / 32);
  for (uint32_t i = blockIdx.y * (blockDim.x / 32) + threadIdx.x / 32; i < m; i += warps) {
    const int32_t sc = lane < kSeedAA ? p32[lane * s32 + i] : INT32_MIN;
    uint32_t place = 0;
#pragma unroll
    for (int a = 0; a < kSeedAA; ++a) {
      const int32_t o = __shfl_sync(0xFFFFFFFFu, sc, a);
      place += o > sc || (o == sc && a < static_cast<int>(lane)) ? 1u : 0u;
    }
    if (lane < kSeedAA) {
      SeedRow& r = rows[row0[qi] + i];
      r.sc[place] = sc;
      r.res[place] = static_cast<uint8_t>(lane);
    }
  }
}

struct SeedQ {
  const uint32_t* qids;
  const uint32_t* woff;  // first window of each query, n_q + 1 entries
  const uint32_t* row0;  // first sorted row of each query
  const uint8_t* res;    // residues of sequence queries (NULL: profile queries)
  const SeedRow* rows;
  uint32_t n_q;
  uint32_t n_win;
  int32_t thr;
  uint32_t cap;
  uint32_t exact;  // add the query's own k-mer
};

__device__ __forceinline__ void seed_window_of(const SeedQ& Q, uint32_t wi, uint32_t& qi, uint32_t& start) {
  uint32_t lo = 0, hi = Q.n_q;  // last qi with woff[qi] <= wi
  while (hi - lo > 1) {
    const uint32_t mid = (lo + hi) / 2;
    if (Q.woff[mid] <= wi) lo = mid; else hi = mid;
  }
  qi = lo;
  start = wi - Q.woff[lo];
}

// Eligibility, exact code and the window's sorted rows (pointers into Q.rows).
__device__ __forceinline__ bool seed_window_rows(const SeedQ& Q, const SeedPat& P, uint32_t qi, uint32_t start,
                                                 const SeedRow** wr, uint32_t& exact) {
  const uint32_t base = Q.row0[qi] + start;
  uint32_t e = 0;
  for (uint32_t i = 0; i < P.w; ++i) {
    if (Q.res) {
      const uint32_t r = Q.res[base + P.offs[i]];
      if (r >= kSeedAA) return false;
      e = e * kSeedAA + r;
    }
    wr[i] = Q.rows + base + P.offs[i];
  }
  exact = e;
  return true;
}

// A window's sorted rows and its suffix maxima in shared memory, by one warp: smax[i] = the best sum of rows i .. w-1.
struct SeedWinRows {
  int32_t sc[kSeedMaxW][kSeedAA];
  uint8_t res[kSeedMaxW][kSeedAA];
  int32_t smax[kSeedMaxW + 1];
};
__device__ __forceinline__ void seed_load_rows(const SeedPat& P, const SeedRow* const* wr, SeedWinRows& o) {
  const uint32_t lane = threadIdx.x & 31;
  for (uint32_t i = 0; i < P.w; ++i)
    if (lane < kSeedAA) {
      o.sc[i][lane] = wr[i]->sc[lane];
      o.res[i][lane] = wr[i]->res[lane];
    }
  __syncwarp();
  if (lane == 0) {
    o.smax[P.w] = 0;
    for (int i = static_cast<int>(P.w) - 1; i >= 0; --i) o.smax[i] = o.smax[i + 1] + o.sc[i][0];
  }
  __syncwarp();
}

// One warp (a CTA) per window: the histogram of the partial sums that can still reach the threshold, row by row, its
// (sum, residue) pairs spread over the lanes with shared-memory atomics.  One thread per window kept both histograms
// in local memory and took 86 us for a lone query of 257 windows, the latency of one thread's chain.
__global__ void __launch_bounds__(32) seed_count_kernel(SeedQ Q, SeedPat P, uint32_t* slots, SeedWin* win,
                                                        SeedStatsDev* st) {
  __shared__ SeedWinRows W;
  __shared__ uint32_t hist[2][kSeedMaxBins];
  unsigned long long n_skip = 0, n_cap = 0, n_err = 0;
  const uint32_t lane = threadIdx.x;
  for (uint32_t wi = blockIdx.x; wi <= Q.n_win; wi += gridDim.x) {
    uint32_t n_slots = 0;
    if (wi < Q.n_win) {
      uint32_t qi, start, exact;
      seed_window_of(Q, wi, qi, start);
      const SeedRow* wr[kSeedMaxW];
      SeedWin wv{INT32_MIN, 0};
      if (!seed_window_rows(Q, P, qi, start, wr, exact)) {
        ++n_skip;
      } else {
        seed_load_rows(P, wr, W);
        uint32_t count = 0;
        if (W.smax[0] >= Q.thr && Q.cap > 0) {
          int32_t lo = 0, hi = 0;
          uint32_t *dist = hist[0], *next = hist[1];
          if (lane == 0) dist[0] = 1;
          __syncwarp();
          bool ok = true;
          for (uint32_t i = 0; i < P.w; ++i) {
            const int32_t nhi = hi + W.sc[i][0];
            const int32_t nlo = max(lo + W.sc[i][kSeedAA - 1], Q.thr - W.smax[i + 1]);
            if (nhi - nlo + 1 > kSeedMaxBins) {
              ok = false;
              break;
            }
            for (int32_t b = lane; b <= nhi - nlo; b += 32) next[b] = 0;
            __syncwarp();
            const int32_t items = (hi - lo + 1) * kSeedAA;
            for (int32_t x = lane; x < items; x += 32) {
              const int32_t off = x / kSeedAA;
              const uint32_t cnt = dist[off];
              const int32_t t = lo + off + W.sc[i][x - off * kSeedAA];
              if (cnt && t >= nlo) atomicAdd(&next[t - nlo], cnt);
            }
            __syncwarp();
            uint32_t* x = dist;
            dist = next;
            next = x;
            lo = nlo;
            hi = nhi;
          }
          if (!ok) {
            ++n_err;
          } else {
            for (int32_t b = lane; b <= hi - lo; b += 32) count += dist[b];
            count = __reduce_add_sync(0xFFFFFFFFu, count);
            if (count > Q.cap) {  // the boundary score, 32 bins at a time from the top
              uint32_t above = 0;
              int32_t top = hi;
              for (;; top -= 32) {
                const int32_t t = top - static_cast<int32_t>(lane);
                const uint32_t cnt = t >= lo ? dist[t - lo] : 0u;
                uint32_t incl = cnt;
#pragma unroll
                for (int o = 1; o < 32; o <<= 1) {
                  const uint32_t y = __shfl_up_sync(0xFFFFFFFFu, incl, o);
                  if (lane >= o) incl += y;
                }
                const uint32_t hit = __ballot_sync(0xFFFFFFFFu, t <= lo || above + incl >= Q.cap);
                if (hit) {
                  const int src = __ffs(hit) - 1;
                  wv.tstar = top - src;
                  wv.need = Q.cap - (above + __shfl_sync(0xFFFFFFFFu, incl - cnt, src));
                  break;
                }
                above += __shfl_sync(0xFFFFFFFFu, incl, 31);
              }
              count = Q.cap;
              ++n_cap;
            }
          }
        }
        n_slots = count + (Q.exact ? 1u : 0u);
        __syncwarp();  // the shared rows and histograms are free for the next window
      }
      if (lane == 0) win[wi] = wv;
    }
    if (lane == 0) slots[wi] = n_slots;
  }
  if (lane == 0) {
    if (n_skip) atomicAdd(&st->windows_skipped, n_skip);
    if (n_cap) atomicAdd(&st->windows_at_cap, n_cap);
    if (n_err) atomicAdd(&st->errors, n_err);
  }
}

// The kept k-mers of each window, one warp (a CTA) per window, level by level: the nodes of a level are the prefixes
// that can still reach the boundary, in rank-lexicographic order, and a node's children are the first ranks of its
// row.  Those that can exceed the boundary score are all kept (each leads to a k-mer above it, so there are at most
// as many as such k-mers); of those that can only reach it, the first `need` in order (each leads to a tie, and
// only the first `need` ties are kept), so a level never holds more than the cap.  Positions come from warp scans,
// and the children of 32 nodes are written 32 at a time whatever their numbers, so a window costs its k-mers over
// the lanes.  The set kept is the depth-first walk's (seed_emit_kernel), in its order.  One thread per window took
// 720 us for a lone query (two CTAs, each thread walking up to 512 k-mers) and 1.38 ms for 150 queries.
constexpr uint32_t kSeedWarpCap = 4096;  // cap of the warp form: two levels of nodes in shared memory

__global__ void __launch_bounds__(32) seed_emit_warp_kernel(SeedQ Q, SeedPat P, const uint32_t* soff,
                                                            const SeedWin* win, SeedSeed* seeds, SeedStatsDev* st) {
  extern __shared__ int2 nodes[];  // [2][cap]: (partial sum, code)
  __shared__ SeedWinRows W;
  constexpr uint32_t FULL = 0xFFFFFFFFu;
  unsigned long long n_gen = 0, n_exact = 0, n_err = 0;
  const uint32_t lane = threadIdx.x;
  for (uint32_t wi = blockIdx.x; wi < Q.n_win; wi += gridDim.x) {
    const uint32_t o0 = soff[wi], o1 = soff[wi + 1];
    if (o1 == o0) continue;
    uint32_t qi, start, exact;
    seed_window_of(Q, wi, qi, start);
    const SeedRow* wr[kSeedMaxW];
    seed_window_rows(Q, P, qi, start, wr, exact);
    const SeedWin wv = win[wi];
    const uint32_t n_kmers = o1 - o0 - (Q.exact ? 1u : 0u);
    bool have_exact = false;
    uint32_t n = 0;
    if (n_kmers > 0) {
      seed_load_rows(P, wr, W);
      const bool capped = wv.tstar != INT32_MIN;
      const int32_t above_from = capped ? wv.tstar + 1 : Q.thr;  // sums from here on are kept whatever their order
      const int32_t from = capped && wv.need ? wv.tstar : above_from;
      int2 *cur = nodes, *nxt = nodes + Q.cap;
      if (lane == 0) cur[0] = make_int2(0, 0);
      __syncwarp();
      uint32_t n_cur = 1;
      for (uint32_t d = 0; d < P.w; ++d) {
        const bool leaf = d + 1 == P.w;
        const int32_t rest = W.smax[d + 1];
        uint32_t n_out = 0, ties = 0;  // children written, ties met
        for (uint32_t c0 = 0; c0 < n_cur; c0 += 32) {
          int2 nd = make_int2(0, 0);
          uint32_t above = 0, all = 0;  // children that can exceed the boundary, that can reach it
          if (c0 + lane < n_cur) {
            nd = cur[c0 + lane];
            // scores descend: the number of ranks whose sum reaches a bound
            auto reach = [&](int32_t bound) {
              uint32_t l = 0, h = kSeedAA;  // ranks below l reach it, ranks from h do not
              while (l < h) {
                const uint32_t mid = (l + h) >> 1;
                if (nd.x + W.sc[d][mid] + rest >= bound) l = mid + 1; else h = mid;
              }
              return l;
            };
            above = reach(above_from);
            all = from == above_from ? above : reach(from);
          }
          uint32_t tie = all - above, tincl = tie;
#pragma unroll
          for (int o = 1; o < 32; o <<= 1) {
            const uint32_t y = __shfl_up_sync(FULL, tincl, o);
            if (lane >= o) tincl += y;
          }
          const uint32_t tbefore = ties + tincl - tie;
          tie = tbefore >= wv.need ? 0u : min(tie, wv.need - tbefore);
          ties += __shfl_sync(FULL, tincl, 31);
          uint32_t incl = above + tie;
#pragma unroll
          for (int o = 1; o < 32; o <<= 1) {
            const uint32_t y = __shfl_up_sync(FULL, incl, o);
            if (lane >= o) incl += y;
          }
          const uint32_t excl = incl - (above + tie);
          const uint32_t total = __shfl_sync(FULL, incl, 31);
          for (uint32_t k0 = 0; k0 < total; k0 += 32) {  // every lane runs every round (shuffles)
            const uint32_t k = k0 + lane;
            uint32_t j = 0;  // last lane whose children begin at or before k
#pragma unroll
            for (int step = 16; step > 0; step >>= 1) {
              const uint32_t oc = __shfl_sync(FULL, excl, (j + step) & 31);
              if (j + step < 32 && oc <= k) j += step;
            }
            const uint32_t r = k - __shfl_sync(FULL, excl, j);
            const int32_t part = __shfl_sync(FULL, nd.x, j);
            const uint32_t code = static_cast<uint32_t>(__shfl_sync(FULL, nd.y, j));
            bool same = false;
            if (k < total) {
              const uint32_t cc = code * kSeedAA + W.res[d][r];
              const uint32_t at = n_out + k;
              if (leaf) {
                if (at < n_kmers) seeds[o0 + at] = SeedSeed{cc, wi};
                same = cc == exact;
              } else if (at < Q.cap) {
                nxt[at] = make_int2(part + W.sc[d][r], static_cast<int>(cc));
              }
            }
            if (leaf) have_exact |= __any_sync(FULL, same);
          }
          n_out += total;
        }
        __syncwarp();
        int2* x = cur;
        cur = nxt;
        nxt = x;
        n_cur = min(n_out, Q.cap);
        n = n_out;
      }
      n_err += n != n_kmers;
      n_gen += n;
      __syncwarp();  // the shared rows and nodes are free for the next window
    }
    if (Q.exact) {
      if (lane == 0) seeds[o0 + n_kmers] = SeedSeed{have_exact ? kSeedNone : exact, wi};
      n_exact += have_exact ? 0 : 1;
      n_gen += have_exact ? 0 : 1;
    }
  }
  if (lane == 0) {
    if (n_gen) atomicAdd(&st->kmers_generated, n_gen);
    if (n_exact) atomicAdd(&st->exact_seeds_added, n_exact);
    if (n_err) atomicAdd(&st->errors, n_err);
  }
}

// The kept k-mers of each window in rank-lexicographic depth-first order, one thread per window: for caps whose levels
// do not fit shared memory (seed_emit_warp_kernel).
__global__ void __launch_bounds__(128) seed_emit_kernel(SeedQ Q, SeedPat P, const uint32_t* soff, const SeedWin* win,
                                                        SeedSeed* seeds, SeedStatsDev* st) {
  unsigned long long n_gen = 0, n_exact = 0, n_err = 0;
  for (uint32_t wi = blockIdx.x * blockDim.x + threadIdx.x; wi < Q.n_win; wi += gridDim.x * blockDim.x) {
    const uint32_t o0 = soff[wi], o1 = soff[wi + 1];
    if (o1 == o0) continue;
    uint32_t qi, start, exact;
    seed_window_of(Q, wi, qi, start);
    const SeedRow* wr[kSeedMaxW];
    seed_window_rows(Q, P, qi, start, wr, exact);
    const SeedWin wv = win[wi];
    const uint32_t w = P.w, last = w - 1;
    int32_t smax[kSeedMaxW + 1];
    smax[w] = 0;
    for (int i = static_cast<int>(w) - 1; i >= 0; --i) smax[i] = smax[i + 1] + wr[i]->sc[0];
    const bool capped = wv.tstar != INT32_MIN;
    int32_t thr = capped ? (wv.need ? wv.tstar : wv.tstar + 1) : Q.thr;
    uint32_t ties = wv.need;
    uint32_t n = 0;
    bool have_exact = false;
    const uint32_t n_kmers = o1 - o0 - (Q.exact ? 1u : 0u);
    if (n_kmers > 0) {
      uint32_t rank[kSeedMaxW], code[kSeedMaxW + 1];
      int32_t part[kSeedMaxW + 1];
      part[0] = 0;
      code[0] = 0;
      rank[0] = 0;
      uint32_t d = 0;
      for (;;) {
        if (d == last) {
          const int32_t bs = part[last];
          const uint32_t bc = code[last] * kSeedAA;
          for (int a = 0; a < kSeedAA; ++a) {
            const int32_t ns = bs + wr[last]->sc[a];
            if (ns < thr) break;
            const uint32_t cc = bc + wr[last]->res[a];
            if (n < n_kmers) seeds[o0 + n] = SeedSeed{cc, wi};  // n == n_kmers at the end (checked below)
            ++n;
            have_exact |= cc == exact;
            if (capped && ns == wv.tstar && --ties == 0) thr = wv.tstar + 1;
          }
          if (last == 0) break;
          d = last - 1;
          ++rank[d];
          continue;
        }
        const uint32_t r = rank[d];
        if (r < kSeedAA) {
          const int32_t ns = part[d] + wr[d]->sc[r];
          if (ns + smax[d + 1] >= thr) {
            part[d + 1] = ns;
            code[d + 1] = code[d] * kSeedAA + wr[d]->res[r];
            ++d;
            rank[d] = 0;
            continue;
          }
        }
        if (d == 0) break;
        --d;
        ++rank[d];
      }
    }
    n_err += n != n_kmers;
    n_gen += n;
    if (Q.exact) {
      if (!have_exact) {
        seeds[o0 + n_kmers] = SeedSeed{exact, wi};
        ++n_exact;
        ++n_gen;
      } else {
        seeds[o0 + n_kmers] = SeedSeed{kSeedNone, wi};
      }
    }
  }
  gate_flush(&st->kmers_generated, n_gen);
  gate_flush(&st->exact_seeds_added, n_exact);
  gate_flush(&st->errors, n_err);
}

// Posting count of each seed (0 for an unused slot, an empty code, or a code
// above max_seed_occ); n_seeds + 1 entries, the last 0.
__global__ void __launch_bounds__(256) seed_post_count_kernel(const SeedSeed* seeds, uint32_t n_seeds,
                                                              const uint32_t* off, uint32_t occ_cap, uint32_t* cnt,
                                                              SeedStatsDev* st) {
  unsigned long long n_seed = 0, n_post = 0, n_over = 0, n_skip = 0;
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i <= n_seeds; i += gridDim.x * blockDim.x) {
    uint32_t len = 0;
    if (i < n_seeds && seeds[i].code != kSeedNone) {
      const uint32_t c = seeds[i].code;
      len = off[c + 1] - off[c];
      if (len > 0 && occ_cap > 0 && len > occ_cap) {
        ++n_over;
        n_skip += len;
        len = 0;
      } else if (len > 0) {
        ++n_seed;
        n_post += len;
      }
    }
    cnt[i] = len;
  }
  gate_flush_block(&st->seeds, n_seed);
  gate_flush_block(&st->postings_visited, n_post);
  gate_flush_block(&st->seeds_over_occ_cap, n_over);
  gate_flush_block(&st->postings_skipped_occ, n_skip);
}

// One hit per posting.  A warp takes 32 consecutive seeds, whose hits are one
// contiguous range of the output; lane k writes output positions k, k + 32, ...
// and finds the seed of each by a binary search over the 32 seeds' offsets held
// in the lanes, so reads of the postings and writes of the hits are coalesced
// whatever the list lengths.  Hits that only the evidence stage reads are
// written as its sort keys: 8 bytes for 16, and no pass that makes keys of them
// (a posting lies inside its target, so none is rejected).
struct SeedHitRecs {
  GateSeedHit* hits;
  __device__ __forceinline__ void put(uint32_t k, uint32_t query, uint32_t target, int32_t diag, uint32_t qpos) const {
    hits[k] = GateSeedHit{query, target, diag, qpos};
  }
};
struct SeedHitKeys {
  uint64_t* keys;
  GateConf g;
  __device__ __forceinline__ void put(uint32_t k, uint32_t query, uint32_t target, int32_t diag, uint32_t qpos) const {
    keys[k] = gate_key(query, target, diag, qpos, g);
  }
};
template <typename OUT>
__global__ void __launch_bounds__(256) seed_hits_kernel(SeedQ Q, const SeedSeed* seeds, uint32_t n_seeds,
                                                        const uint32_t* cnt, const uint32_t* hoff, const uint32_t* off,
                                                        const SeedPost* post, const OUT out) {
  const uint32_t lane = threadIdx.x & 31;
  const uint32_t n_groups = (n_seeds + 31) / 32;
  for (uint32_t g = (blockIdx.x * blockDim.x + threadIdx.x) / 32; g < n_groups; g += (gridDim.x * blockDim.x) / 32) {
    const uint32_t s = g * 32 + lane;
    // this lane's seed: first output position, posting start, query and position
    uint32_t o = 0, pstart = 0, q = 0, start = 0;
    if (s < n_seeds) {
      o = hoff[s];
      if (cnt[s]) {
        const SeedSeed sd = seeds[s];
        uint32_t qi;
        seed_window_of(Q, sd.window, qi, start);
        q = Q.qids[qi];
        pstart = off[sd.code];
      }
    }
    const uint32_t last = min(n_seeds, g * 32 + 32);
    const uint32_t o_begin = __shfl_sync(0xFFFFFFFFu, o, 0);
    const uint32_t o_end = hoff[last];
    for (uint32_t base = o_begin; base < o_end; base += 32) {  // every lane runs every round (shuffles)
      const uint32_t k = base + lane;
      const bool live = k < o_end;
      // last lane j with offset <= k (lanes past the group's seeds are never chosen)
      uint32_t j = 0;
#pragma unroll
      for (int step = 16; step > 0; step >>= 1) {
        const uint32_t cand = j + step;
        const uint32_t oc = __shfl_sync(0xFFFFFFFFu, o, cand & 31);
        if (cand < last - g * 32 && oc <= k) j = cand;
      }
      const uint32_t oj = __shfl_sync(0xFFFFFFFFu, o, j);
      const uint32_t pj = __shfl_sync(0xFFFFFFFFu, pstart, j);
      const uint32_t qj = __shfl_sync(0xFFFFFFFFu, q, j);
      const uint32_t sj = __shfl_sync(0xFFFFFFFFu, start, j);
      if (live) {
        const SeedPost ps = post[pj + (k - oj)];
        out.put(k, qj, ps.target, static_cast<int32_t>(ps.tpos) - static_cast<int32_t>(sj), sj);
      }
    }
  }
}

}  // namespace st
