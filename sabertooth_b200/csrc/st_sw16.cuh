// Packed 16-bit Smith-Waterman-Gotoh score kernel (the fast path of the
// reference's QueryProfile::sw_score_with, src/simd.rs:252-292).
//
// Work layout.  A group of G lanes of one warp scores TWO targets of the same
// query at once, one per 16-bit half of every register (s16x2).  Lane l of the
// group owns R consecutive query rows; the targets stream through the group as
// a wavefront, C columns per step (lane l works on columns [c, c+C) while lane
// l-1 works on [c+C, c+2C)), so per step each lane receives from the lane
// above, by __shfl_up_sync, a control word, the residue codes of its C
// columns, and the bottom-row H and the F entering its first row for each of
// them.  Queries longer than G*R rows are scored in passes over the targets;
// the bottom row of a pass goes through a per-group scratch line in global
// memory and comes back into lane 0 for the next pass.
//
// Streaming.  A warp pulls warp tasks (64/G targets of the query, two per
// group, padded to a common length) one after another and feeds them into the
// wavefront back to back: lane 0 starts the next task while the lower lanes
// finish the previous one, so the G-1 step ramp is paid once per query, not
// per task.  The control word that travels with the columns tells each lane
// the column, the pass, when to reset its state (first column of a pass) and
// when a task ends; at that point every lane folds its running maximum into
// the task's slot in shared memory, and the last lane of the group, which
// finishes the task last, writes the two scores.  The next task is claimed and
// its slot records loaded one task ahead, so the loads are off the critical
// path.
//
// Recurrence per cell: Gotoh's (the reference's scalar kernel,
// src/simd.rs:361-374), with both gap states opened from the match state
//   t = max(Hdiag + S, E, 0);  H = max(t, F)
//   E' = max(E - x, t - open)        (E of the next column)
//   F' = max(F - x, t - open)        (F of the next row),  x = min(open, extend)
// Every H equals the literal recurrence's.  Reopening a gap out of itself
// costs open where extending costs extend, so opening from H instead of t only
// matters for open < extend, which x covers; a gap in one sequence directly
// followed by one in the other scores the same in either order, and the order
// E then F is kept (t holds E).  The maximum is always reached in some t (a gap
// never raises it), so `best` follows t.  With H out of the F chain the serial
// part of a row is one operation (F') instead of three; what bounds the kernel
// is the ALU pipe: 5.5 operations a cell pair (t, H, half a three-way best, E',
// F', prmt), the packed add runs beside them on the multiply pipe.  Measured, B200:
// the 1.2 M-pair PSSM plan 24.93 -> 24.61 ms, 4 M exhaustive pairs 75.6 -> 74.1 ms, one
// 250 x 300 call 88.7 -> 83.2 us.  Scores by byte dot products on the multiply
// pipe instead of prmt measured no faster (6.3 against 6.4 T cells/s in a bare cell
// loop: the third register operand of both pipes' instructions is what limits then).
//
// Teams.  In the team form a CTA's warps share one warp task and run its passes
// side by side: warp w takes passes w, w + 8, ..., each some 36 steps behind the pass
// above it, whose feeder publishes the columns of its boundary line in a counter.
// It is for batches that a query of many rows would otherwise keep waiting: the
// wavefront of 2,000 rows x 900 columns is 510 steps of 32 x 8 rows instead of 480 of
// 32 x 32 (938 against 1,932 cycles each) or 1,830 of 32 x 8.
//
// End cells.  In the end modes a column's maximum is compared with a threshold
// before anything else is done: the best score seen by this lane or by the lanes
// above it (their g travels with the columns), less one, as an equal score may
// come first by its column.  Only a column above it looks for the row and
// updates the lane's optimum, ordered by score, column, row; the fold takes the
// first over the lanes.  The reverse pass knows its score, so only the optimum
// itself passes its threshold; it stages the query backwards, reads the target
// backwards from the end cell, and masks the rows before the prefix to score 0,
// which leaves H = 0 and the gap states of a first row, the prefix's border.
// 4,000 spans of 280 x 280 cells took 4.0 ms with one warp a pair in 32 bits.
//
// Exactness.  The adds wrap instead of saturating.  If no t anywhere exceeds
// T = 32767 - max(0, max score), no sum can leave the int16 range (E, F >=
// -open-extend, S is int8), so the result is exact; otherwise the first t
// above T was itself computed exactly and the pair is flagged for the exact
// 32-bit kernel.  Rows past the query and columns past a target score 0, which
// cannot raise the maximum when open, extend >= 0 (the only gap costs this
// kernel is used for).
#pragma once
#include "st_common.cuh"

namespace st {

struct Sw16CtaTask {
  uint32_t query;
  uint32_t wt_begin;
  uint32_t wt_end;
  uint32_t m_pad;  // P * G * R rows staged in shared memory
};

struct Sw16WarpTask {
  uint32_t slot_begin;  // 64/G consecutive slot records, two per group
  uint32_t ncols;       // columns streamed per pass: multiple of 4, >= 32 (>= C*G with several passes)
};

// One target of a warp task: everything lane 0 needs, in one 16-byte load.
struct Sw16Slot {
  uint32_t pair;    // pair index, kNoPair for an empty slot
  uint32_t toff16;  // database arena offset of the target / 16
  uint32_t tlen16;  // target length rounded up to 16 (readable bytes)
  uint32_t tlen;    // target length
};

struct Sw16Params {
  const uint8_t* arena;  // padded residue arena
  DeviceProfiles prof;
  const Sw16CtaTask* cta_tasks;
  uint32_t n_cta_tasks;
  const Sw16WarpTask* warp_tasks;
  const Sw16Slot* slots;
  int32_t* scores;        // per pair
  uint32_t* kernels;      // per pair (may be null)
  uint32_t* ovf_count;    // pairs above the 16-bit headroom
  uint32_t* ovf_pairs;
  uint32_t* work_counter; // next CTA task (reset before each launch)
  uint2* scratch;         // pass boundary rows, scratch_stride entries per group
  uint32_t scratch_stride;
  int32_t open, ext;
  uint32_t team_spins;    // team form: polls of a producer's count before a team gives its pair up
  // end-cell modes: end cell (query, target) of each pair, -1 for a zero score; in the reverse mode the end of
  // the reversed prefix [0, rev_q] x [0, rev_t] whose forward score is rev_score
  int32_t* end_q = nullptr;
  int32_t* end_t = nullptr;
  const int32_t* rev_q = nullptr;
  const int32_t* rev_t = nullptr;
  const int32_t* rev_score = nullptr;
};

// What a pass reports: the score; the score and its end cell, the first optimum in column-major order
// (src/simd.rs:375-381); or the end cell of the reversed prefixes (the start search of align_canonical,
// src/align.rs:848-866), whose score is known.
enum Sw16Mode { kSw16Score = 0, kSw16End = 1, kSw16RevEnd = 2 };

constexpr uint32_t kNoPair = 0xFFFFFFFFu;

// control word: events, with the pass (bits 16-23) and the task slot (24-26) they belong to
constexpr uint32_t kCtlLast = 1u << 27;   // last step of the task
constexpr uint32_t kCtlFirst = 1u << 28;  // first step of a pass
constexpr uint32_t kCtlMore = 1u << 29;   // a pass that is not the last: its bottom row is kept
constexpr uint32_t kMaxPasses16 = 256;    // passes that bits 16-23 can name; the planners admit no more
constexpr int kSlotRing = 8;
constexpr uint32_t kTeamSpins = 1u << 22;  // the default of Sw16Params::team_spins

template <int G, int R, int C>
struct Sw16Tile {
  static_assert(G == 4 || G == 8 || G == 16 || G == 32, "group size");
  static_assert(R % 4 == 0 && R >= 8 && R <= 32, "rows per lane");
  static_assert(C == 2 || C == 4, "columns per step");
  static constexpr int kGroups = 32 / G;
  static constexpr int kSlots = 2 * kGroups;
  static constexpr int kWords = R / 4;
};

// This lane's R profile bytes of one residue row (R/4 words); the lane's
// first row is R-byte aligned, so the widest vector that divides R is used.
template <int R>
__device__ __forceinline__ void load_rows8(const int8_t* p, uint32_t (&w)[R / 4]) {
  if constexpr (R % 16 == 0) {
#pragma unroll
    for (int v = 0; v < R / 16; ++v) {
      const uint4 x = *reinterpret_cast<const uint4*>(p + 16 * v);
      w[4 * v + 0] = x.x;
      w[4 * v + 1] = x.y;
      w[4 * v + 2] = x.z;
      w[4 * v + 3] = x.w;
    }
  } else if constexpr (R % 8 == 0) {
#pragma unroll
    for (int v = 0; v < R / 8; ++v) {
      const uint2 x = *reinterpret_cast<const uint2*>(p + 8 * v);
      w[2 * v + 0] = x.x;
      w[2 * v + 1] = x.y;
    }
  } else {
#pragma unroll
    for (int v = 0; v < R / 4; ++v) w[v] = *reinterpret_cast<const uint32_t*>(p + 4 * v);
  }
}

// C residue codes of a target starting at column c (c is a multiple of C), or sentinels past its end or without
// `on`.  A predicated load: the lanes that do not feed the stream pass it without a branch.
template <int C>
__device__ __forceinline__ uint32_t load_codes(bool on, const uint8_t* t, uint32_t len16, int c) {
  uint32_t v = 0x15151515u & (C == 4 ? 0xFFFFFFFFu : 0xFFFFu);
  const uint32_t p = on && static_cast<uint32_t>(c) < len16;
  if constexpr (C == 4)
    asm volatile("{ .reg .pred q; setp.ne.u32 q, %2, 0; @q ld.global.nc.u32 %0, [%1]; }" : "+r"(v) : "l"(t + c), "r"(p));
  else
    asm volatile("{ .reg .pred q; setp.ne.u32 q, %2, 0; @q ld.global.nc.u16 %0, [%1]; }" : "+r"(v) : "l"(t + c), "r"(p));
  return v;
}

// Four residues of a target read backwards from position last: positions last - c .. last - c - 3 (sentinels
// below position 0), from two aligned words.
__device__ __forceinline__ uint32_t load_codes_rev(const uint8_t* t, int last, int c) {
  const int p = last - c;
  if (p < 0) return 0x15151515u;
  const uint32_t* w = reinterpret_cast<const uint32_t*>(t) + (p >> 2);
  const uint32_t hi = __ldg(w), lo = p >= 4 ? __ldg(w - 1) : 0x15151515u;
  const uint32_t s = static_cast<uint32_t>(p & 3);
  return __byte_perm(lo, hi, 0x1234u + s * 0x1111u);  // bytes s + 4, s + 3, s + 2, s + 1 of the eight
}

// acc + (byte j of bytes) * mul: the 16-bit x byte dot product with mul in the half that meets byte j
// (bits 16-31 for odd j) and zero in the other.
__device__ __forceinline__ uint32_t dot_byte(int j, uint32_t mul, uint32_t bytes, uint32_t acc) {
  uint32_t d;
  if (j < 2)
    asm("dp2a.lo.u32.u32 %0, %1, %2, %3;" : "=r"(d) : "r"(mul), "r"(bytes), "r"(acc));
  else
    asm("dp2a.hi.u32.u32 %0, %1, %2, %3;" : "=r"(d) : "r"(mul), "r"(bytes), "r"(acc));
  return d;
}

// (H, F) of C columns of the boundary line, loaded or stored when `on` (predicated, as load_codes).
template <int C>
__device__ __forceinline__ void load_bnd(bool on, const uint2* b, uint32_t (&h)[C], uint32_t (&f)[C]) {
  static_assert(C % 2 == 0, "whole vectors");
  const uint32_t p = on;
#pragma unroll
  for (int j = 0; j < C; j += 2)
    asm volatile("{ .reg .pred q; setp.ne.u32 q, %5, 0; @q ld.global.v4.u32 {%0, %1, %2, %3}, [%4]; }"
                 : "+r"(h[j]), "+r"(f[j]), "+r"(h[j + 1]), "+r"(f[j + 1])
                 : "l"(b + j), "r"(p)
                 : "memory");
}
template <int C>
__device__ __forceinline__ void store_bnd(bool on, uint2* b, const uint32_t (&h)[C], const uint32_t (&f)[C]) {
  const uint32_t p = on;
#pragma unroll
  for (int j = 0; j < C; j += 2)
    asm volatile("{ .reg .pred q; setp.ne.u32 q, %5, 0; @q st.global.v4.u32 [%4], {%0, %1, %2, %3}; }" ::"r"(h[j]),
                 "r"(f[j]), "r"(h[j + 1]), "r"(f[j + 1]), "l"(b + j), "r"(p)
                 : "memory");
}

// Per-group view of a warp task's two targets (meaningful in the group's lane 0).
struct Sw16Pair2 {
  const uint8_t* tA;
  const uint8_t* tB;
  uint32_t lenA, lenB;  // reverse mode: residues of the prefix
  uint32_t pA, pB;
  int32_t sA, sB;       // reverse mode: the forward scores
  uint32_t offA, offB;  // and the rows of the reversed query before the prefix
};

__device__ __forceinline__ Sw16Pair2 load_pair2(const Sw16Params& prm, uint32_t slot_begin, int grp) {
  const uint4 a = __ldg(reinterpret_cast<const uint4*>(prm.slots + slot_begin + 2 * grp));
  const uint4 b = __ldg(reinterpret_cast<const uint4*>(prm.slots + slot_begin + 2 * grp + 1));
  Sw16Pair2 r;
  r.pA = a.x;
  r.pB = b.x;
  r.tA = prm.arena + static_cast<size_t>(a.y) * 16;
  r.tB = prm.arena + static_cast<size_t>(b.y) * 16;
  r.lenA = a.x == kNoPair ? 0u : a.z;
  r.lenB = b.x == kNoPair ? 0u : b.z;
  return r;
}

// The reverse mode's view: the prefix of each half and its score (0: nothing to search, the pair scored 0 or is
// in the 32-bit list).
__device__ __forceinline__ void load_rev(const Sw16Params& prm, uint32_t p, uint32_t m, int32_t thresh, uint32_t& len,
                                         int32_t& score, uint32_t& off) {
  len = 0;
  score = 0;
  off = 0;
  if (p == kNoPair) return;
  const int32_t s = prm.rev_score[p];
  if (s <= 0 || s > thresh) return;
  score = s;
  len = static_cast<uint32_t>(prm.rev_t[p]) + 1;
  off = m - 1 - static_cast<uint32_t>(prm.rev_q[p]);
}

// Bytes of word v (rows 4v .. 4v+3 of a lane) that lie at or past row nz, as a byte mask.
__device__ __forceinline__ uint32_t rows_from(int nz, int v) {
  const int k = nz - 4 * v;
  return k <= 0 ? 0xFFFFFFFFu : (k >= 4 ? 0u : 0xFFFFFFFFu << (8 * k));
}

// Persistent kernel: CTAs pull CTA tasks (one query each) from a global
// counter and stage the query's int8 profile in shared memory; each warp then
// streams the CTA task's warp tasks, its first by its number and the others claimed from a shared counter.
//
// Beside the cells a step costs its 3 + 2C shuffles, the residues' row offsets
// (one dot product each, dot_byte) and the feeder's loads and stores, which are
// predicated; one vote decides whether any lane is at an event or lane 0 near
// the end of its pass, and only then the stream is looked at (a lone warp's
// step spent 160 of 1,140 cycles on resolving 15 branches, now 4).  Registers are
// the other lever: asking for three CTAs of four warps (R >= 28, up to 168
// registers) or three of eight (R = 8) and two of eight otherwise lets the
// profile loads of a column be issued ahead of its rows.  Streamed cells/s of
// single classes on the 1.2 M-pair PSSM batch, before -> after: <8,24> 5.41 -> 5.77 T,
// <16,24> 5.40 -> 5.76, <16,32> 5.13 -> 5.62, <8,16> 4.96 -> 5.33, <8,12> 4.82 -> 5.17; a lone
// warp's step <8,24> 1,756 -> 1,541 cycles, <8,8> 1,050 -> 771.
template <int G, int R, int C, int WARPS, int MODE = kSw16Score, bool TEAM = false>
__global__ void __launch_bounds__(WARPS * 32, WARPS == 4 || (R == 8 && MODE == kSw16Score) ? 3 : 2)
    sw16_kernel(const Sw16Params prm) {
  using Tile = Sw16Tile<G, R, C>;
  constexpr int NG = Tile::kGroups;
  constexpr uint32_t FULL = 0xFFFFFFFFu;
  extern __shared__ __align__(16) int8_t prof_s[];
  __shared__ uint32_t s_task, s_next;
  __shared__ int32_t s_best[WARPS][NG][kSlotRing][2];
  __shared__ uint32_t s_pair[WARPS][NG][kSlotRing][2];
  constexpr bool kEnds = MODE != kSw16Score;
  // end-cell modes: (score, inverted column and row) of a task's two targets, largest first; the reverse mode's
  // (forward score, rows before the prefix)
  __shared__ unsigned long long s_end[kEnds ? WARPS : 1][kEnds ? NG : 1][kSlotRing][2];
  __shared__ int2 s_rev[MODE == kSw16RevEnd ? WARPS : 1][MODE == kSw16RevEnd ? NG : 1][kSlotRing][2];

  // team form: a column count per warp, that of the boundary columns it has published; and whether a wait ran out
  __shared__ volatile uint32_t s_prog[TEAM ? WARPS : 1];
  __shared__ volatile uint32_t s_fail;
  static_assert(!TEAM || (G == 32 && MODE == kSw16Score), "a team's warps are whole groups");

  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  const int gl = lane % G;
  const int grp = lane / G;
  const int own = TEAM ? 0 : warp;  // whose slots this warp's tasks use
  uint2* bnd = prm.scratch + static_cast<size_t>((blockIdx.x * WARPS + warp) * NG + grp) * prm.scratch_stride;
  const uint32_t MOPEN = pk_splat(-prm.open);
  const uint32_t MEXT = pk_splat(-min(prm.ext, prm.open));
  const uint32_t E0 = MOPEN;  // E of the first column: max(0 - open, -inf)
  const uint32_t F0 = MOPEN;  // F of the first row
  const uint32_t SENTW = 0x15151515u;

  for (;;) {
    if (threadIdx.x == 0) s_task = atomicAdd(prm.work_counter, 1u);
    __syncthreads();
    const uint32_t ct = s_task;
    if (ct >= prm.n_cta_tasks) break;
    const Sw16CtaTask task = prm.cta_tasks[ct];
    const uint32_t q = task.query;
    const uint32_t m_pad = task.m_pad;
    const int P = static_cast<int>(m_pad / (G * R));
    const uint32_t m = MODE == kSw16RevEnd ? prm.prof.qlen[q] : 0u;
    {  // stage the profile: 22 residue rows of m_pad int8 scores, zero past the stored stride
      const uint32_t chunks_per_row = m_pad / 16;
      const uint32_t stride = prm.prof.stride8[q];
      const int8_t* src = prm.prof.p8[q];
      for (uint32_t idx = threadIdx.x; idx < kProfRows * chunks_per_row; idx += WARPS * 32) {
        const uint32_t r = idx / chunks_per_row;
        const uint32_t i = (idx - r * chunks_per_row) * 16;
        uint4 v = make_uint4(0, 0, 0, 0);
        if constexpr (MODE == kSw16RevEnd) {  // the query backwards
          int8_t* b = reinterpret_cast<int8_t*>(&v);
#pragma unroll
          for (int k = 0; k < 16; ++k)
            if (i + k < m) b[k] = src[static_cast<size_t>(r) * stride + (m - 1 - i - k)];
        } else {
          if (i < stride) v = *reinterpret_cast<const uint4*>(src + static_cast<size_t>(r) * stride + i);
        }
        *reinterpret_cast<uint4*>(prof_s + static_cast<size_t>(r) * m_pad + i) = v;
      }
    }
    if (threadIdx.x == 0) s_next = task.wt_begin + WARPS;
    if constexpr (TEAM) {
      if (threadIdx.x < WARPS) s_prog[threadIdx.x] = 0;
      if (threadIdx.x == 0) {
        s_fail = 0;
        s_best[0][0][0][0] = 0;
        s_best[0][0][0][1] = 0;
      }
    }
    const int32_t thresh = 32767 - prm.prof.max_score[q];
    __syncthreads();

    // ---- the warp's stream over warp tasks ----
    // The group's last lane (the feeder) tracks lane 0's position in the stream (the same
    // uniform state in every lane), loads the targets' residues and the previous pass's
    // bottom row for lane 0's next step, and leaves them in its outgoing registers: the
    // rotating shuffle then hands lane 0 the stream and every other lane its upper
    // neighbour's outputs.
    const bool feeder = gl == G - 1;
    const int src_lane = (lane & ~(G - 1)) | ((lane - 1) & (G - 1));
    // a warp's first warp task goes by its number, so that a task of few has them on different schedulers and no warp
    // has two while another has none; the others are claimed
    auto claim = [&]() -> uint32_t {
      uint32_t w = 0;
      if (lane == 0) w = atomicAdd(&s_next, 1u);
      return __shfl_sync(FULL, w, 0);
    };
    // a team's warps share the CTA task's one warp task: warp w takes its passes w, w + WARPS, ...
    uint32_t w_cur = __shfl_sync(FULL, task.wt_begin + (TEAM ? 0u : static_cast<uint32_t>(warp)), 0);
    bool have = TEAM ? warp < P : w_cur < task.wt_end;
    if (have) {
    auto load_pairs = [&](uint32_t slot_begin) {
      Sw16Pair2 r = load_pair2(prm, slot_begin, grp);
      if constexpr (MODE == kSw16RevEnd) {
        load_rev(prm, r.pA, m, thresh, r.lenA, r.sA, r.offA);
        load_rev(prm, r.pB, m, thresh, r.lenB, r.sB, r.offB);
      }
      return r;
    };
    // the reverse mode streams the longest prefix of the task, not its longest target (all lanes call it)
    auto clip = [&](Sw16WarpTask& wt, const Sw16Pair2& r) {
      if constexpr (MODE == kSw16RevEnd) {
        const uint32_t len = __reduce_max_sync(FULL, feeder ? max(r.lenA, r.lenB) : 0u);
        const uint32_t least = P > 1 ? (C * G + 15u) & ~15u : 32u;
        wt.ncols = min(wt.ncols, max(least, (len + 3u) & ~3u));
      }
    };
    auto load_step = [&](const uint8_t* t, uint32_t len, int c) -> uint32_t {
      if constexpr (MODE == kSw16RevEnd) return feeder ? load_codes_rev(t, static_cast<int>(len) - 1, c) : SENTW;
      else return load_codes<C>(feeder, t, len, c);
    };
    // a task enters the ring (the group's feeder)
    auto open_slot = [&](int slot, const Sw16Pair2& r) {
      s_pair[own][grp][slot][0] = r.pA;
      s_pair[own][grp][slot][1] = r.pB;
      if constexpr (kEnds) {
        s_end[warp][grp][slot][0] = 0;
        s_end[warp][grp][slot][1] = 0;
        if constexpr (MODE == kSw16RevEnd) {
          s_rev[warp][grp][slot][0] = make_int2(r.sA, static_cast<int>(r.offA));
          s_rev[warp][grp][slot][1] = make_int2(r.sB, static_cast<int>(r.offB));
        }
      } else {
        s_best[own][grp][slot][0] = 0;
        s_best[own][grp][slot][1] = 0;
      }
    };
    Sw16WarpTask wt_cur = prm.warp_tasks[w_cur];
    Sw16Pair2 cur{};
    if (feeder) cur = load_pairs(wt_cur.slot_begin);
    clip(wt_cur, cur);
    uint32_t w_nxt = TEAM ? task.wt_end : claim();
    bool have_nxt = w_nxt < task.wt_end;
    Sw16WarpTask wt_nxt = have_nxt ? prm.warp_tasks[w_nxt] : Sw16WarpTask{0, 0};
    Sw16Pair2 nxt{};
    if (have_nxt && feeder) nxt = load_pairs(wt_nxt.slot_begin);
    if (have_nxt) clip(wt_nxt, nxt);
    if (!TEAM && feeder) open_slot(0, cur);
    // Lane 0's position: column u_col of pass u_pass of task u_seq.  The control word of an ordinary step is
    // u_ctl; the first and the last step of a pass add their events, so an ordinary step takes no decisions
    // beyond one vote (is any lane at an event, or lane 0 within a step of its pass's end).
    constexpr int kPassStep = TEAM ? WARPS : 1;
    int u_col = 0, u_pass = TEAM ? warp : 0, u_seq = 0;
    bool done = false, gap = false;
    int u_end = static_cast<int>(wt_cur.ncols);  // columns of the pass; of the idle steps at the end of the stream
    uint32_t u_ctl = u_pass + 1 < P ? kCtlMore : 0u;
    uint32_t u_last = u_pass + kPassStep < P ? 0u : kCtlLast;  // the event of the pass's last step

    // per-lane wavefront state
    uint32_t Hp[R], E[R];
#pragma unroll
    for (int k = 0; k < R; ++k) {
      Hp[k] = 0;
      E[k] = E0;
    }
    uint32_t best = 0, hup_prev = 0;
    uint32_t row0 = static_cast<uint32_t>(gl * R);  // this lane's first row of its pass
    uint32_t my_col = 0;                            // its column
    const uint32_t mul_lo = m_pad, mul_hi = m_pad << 16;
    // end-cell modes: this lane's first optimum per half as score and column << 16 | row; thr: only a cell above
    // it is looked at; g: the best score of the lanes above and of this one
    int32_t endsA = 0, endsB = 0;
    uint32_t endA = 0, endB = 0, thr = 0, g = 0;
    uint32_t maskA[kEnds ? Tile::kWords : 1], maskB[kEnds ? Tile::kWords : 1];
    if constexpr (MODE == kSw16RevEnd) {
#pragma unroll
      for (int v = 0; v < Tile::kWords; ++v) maskA[v] = maskB[v] = 0xFFFFFFFFu;
    }
    // outgoing registers: a lane's outputs for the lane below (the feeder: lane 0's next inputs)
    uint32_t my_ctl = 0, my_rA = SENTW, my_rB = SENTW;
    uint32_t my_h[C], my_f[C];
#pragma unroll
    for (int j = 0; j < C; ++j) {
      my_h[j] = 0;
      my_f[j] = F0;
    }
    // lane 0's first step: column 0, pass 0 of the first task
    if (feeder) my_ctl = kCtlFirst | u_ctl | (static_cast<uint32_t>(u_pass) << 16);
    my_rA = load_step(cur.tA, cur.lenA, 0);
    my_rB = load_step(cur.tB, cur.lenB, 0);
    // Team form: the boundary of the next step comes from the warp that runs the pass above, once it has published
    // the columns.  The wait is bounded; when it runs out the pair goes to the exact 32-bit kernel instead.
    const uint32_t team_cols = wt_cur.ncols;
    uint32_t seen = 0;     // columns of the producer known to be published
    uint32_t my_base = 0;  // this lane's columns published in earlier passes
    auto team_load = [&]() {
      const int from = (u_pass - 1) % WARPS;
      const uint32_t need = static_cast<uint32_t>((u_pass - 1) / WARPS) * team_cols + u_col + C;
      if (seen < need) {
        for (uint32_t spin = 0; (seen = s_prog[from]) < need && s_fail == 0; ++spin)
          if (spin >= prm.team_spins) s_fail = 1;
        __threadfence_block();
      }
      load_bnd<C>(true, prm.scratch + static_cast<size_t>(blockIdx.x * WARPS + from) * prm.scratch_stride + u_col,
                  my_h, my_f);
    };
    if constexpr (TEAM)
      if (feeder && u_pass > 0) team_load();
    __syncwarp();

    for (;;) {
      // this step's inputs: from the lane above, lane 0 from the feeder
      const uint32_t ctl = __shfl_sync(FULL, my_ctl, src_lane);
      const uint32_t rA = __shfl_sync(FULL, my_rA, src_lane);
      const uint32_t rB = __shfl_sync(FULL, my_rB, src_lane);
      uint32_t h_in[C], f_in[C];
#pragma unroll
      for (int j = 0; j < C; ++j) {
        h_in[j] = __shfl_sync(FULL, my_h[j], src_lane);
        f_in[j] = __shfl_sync(FULL, my_f[j], src_lane);
      }
      uint32_t g_in = 0;
      if constexpr (MODE == kSw16End) g_in = __shfl_sync(FULL, g, src_lane);
      my_ctl = ctl;
      my_rA = rA;
      my_rB = rB;
      // lane 0's next step (uniform across the warp)
      uint32_t n_ctl = u_ctl;
      u_col += C;
      const bool event = __any_sync(FULL, (ctl & (kCtlFirst | kCtlLast)) != 0 || u_col + C >= u_end);
      if (event) {
        if (u_col == u_end) {
          n_ctl = kCtlFirst;
          if (!have) {  // the idle steps are over
            done = true;
          } else if (TEAM && !gap && u_pass + kPassStep < P) {
            gap = true;  // a team's warp finishes and publishes a pass before it may have to wait for its next one
          } else {
            gap = false;
            u_pass += kPassStep;
            if (u_pass >= P) {  // task done: the pre-claimed task becomes current, claim the one after
              u_pass = 0;
              ++u_seq;
              have = have_nxt;
              wt_cur = wt_nxt;
              cur = nxt;
              if (have) {
                if (feeder) open_slot(u_seq & (kSlotRing - 1), cur);
                w_nxt = claim();
                have_nxt = w_nxt < task.wt_end;
                if (have_nxt) {
                  wt_nxt = prm.warp_tasks[w_nxt];
                  if (feeder) nxt = load_pairs(wt_nxt.slot_begin);
                  clip(wt_nxt, nxt);
                }
                u_end = static_cast<int>(wt_cur.ncols);
              }
            }
          }
          u_col = 0;
          if (have && !gap) {
            if constexpr (TEAM) u_end = static_cast<int>(team_cols);
            const uint32_t at = (static_cast<uint32_t>(u_pass) << 16) |
                                (static_cast<uint32_t>(u_seq & (kSlotRing - 1)) << 24);
            u_ctl = u_pass + 1 < P ? kCtlMore : 0u;
            u_last = u_pass + kPassStep < P ? 0u : kCtlLast | at;
            n_ctl |= u_ctl | at;
          } else {  // idle steps until the last lane has finished
            if (!TEAM) cur.lenA = cur.lenB = 0;
            u_ctl = u_last = n_ctl = 0u;
            u_end = (G - 1) * C;
          }
        } else if (u_col + C == u_end) {
          n_ctl |= u_last;
        }
        // first column of a pass: left border H = 0, first-column E
        if (ctl & kCtlFirst) {
#pragma unroll
          for (int k = 0; k < R; ++k) {
            Hp[k] = 0;
            E[k] = E0;
          }
          hup_prev = 0;
          my_col = 0;
          row0 = ((ctl >> 16) & 0xFFu) * (G * R) + gl * R;
          if constexpr (TEAM) my_base = ((ctl >> 16) & 0xFFu) / WARPS * team_cols;
          if constexpr (kEnds) {
            const bool begin = (ctl & 0x00FF0000u) == 0;  // the task's first pass
            if (begin) {
              endsA = endsB = 0;
              endA = endB = 0;
              g = 0;
            }
            if constexpr (MODE == kSw16RevEnd) {
              // only the known score is looked for; the rows before the prefix score 0 (H = 0, as above a query)
              const int slot = static_cast<int>((ctl >> 24) & 7u);
              const int2 a = s_rev[warp][grp][slot][0], b = s_rev[warp][grp][slot][1];
              thr = (a.x > 0 ? static_cast<uint32_t>(a.x - 1) : 32767u) |
                    ((b.x > 0 ? static_cast<uint32_t>(b.x - 1) : 32767u) << 16);
#pragma unroll
              for (int v = 0; v < Tile::kWords; ++v) {
                maskA[v] = rows_from(a.y - static_cast<int>(row0), v);
                maskB[v] = rows_from(b.y - static_cast<int>(row0), v);
              }
            } else {
              // a later pass may reach the same score in an earlier column
              thr = static_cast<uint32_t>(max(endsA - 1, 0)) | (static_cast<uint32_t>(max(endsB - 1, 0)) << 16);
            }
          }
        }
        __syncwarp();
      }
      // the feeder's residues, on their way while this step is computed
      const bool idle = TEAM && (gap || !have);
      const uint32_t nA = load_step(cur.tA, idle ? 0u : cur.lenA, u_col);
      const uint32_t nB = load_step(cur.tB, idle ? 0u : cur.lenB, u_col);
      if constexpr (MODE == kSw16End) {
        if (gl != 0) g = pk_max(g, g_in);
        thr = pk_max(thr, pk_add(g, 0xFFFFFFFFu));  // g - 1: an equal score may come first by its column
      }
#pragma unroll
      for (int j = 0; j < C; ++j) {
        // row0 + residue * m_pad: one 16-bit x byte dot product picks the byte and multiplies it
        const uint32_t oA = dot_byte(j, j & 1 ? mul_hi : mul_lo, rA, row0);
        const uint32_t oB = dot_byte(j, j & 1 ? mul_hi : mul_lo, rB, row0);
        uint32_t wa[Tile::kWords], wb[Tile::kWords];
        load_rows8<R>(prof_s + oA, wa);
        load_rows8<R>(prof_s + oB, wb);
        if constexpr (MODE == kSw16RevEnd) {
#pragma unroll
          for (int v = 0; v < Tile::kWords; ++v) {
            wa[v] &= maskA[v];
            wb[v] &= maskB[v];
          }
        }
        uint32_t hd = j == 0 ? hup_prev : h_in[j - 1];
        uint32_t F = f_in[j];
        uint32_t t_odd = 0;
        if constexpr (kEnds) best = 0;  // the column's
#pragma unroll
        for (int k = 0; k < R; ++k) {
          const uint32_t S = prmt(wa[k >> 2], wb[k >> 2], sel_pair(k & 3));
          const uint32_t t = pk_addmax_relu(hd, S, E[k]);
          const uint32_t To = pk_add(t, MOPEN);
          hd = Hp[k];
          Hp[k] = pk_max(t, F);
          E[k] = pk_addmax(E[k], MEXT, To);
          F = pk_addmax(F, MEXT, To);
          if (k & 1)
            best = pk_max3(best, t_odd, t);
          else
            t_odd = t;
        }
        my_h[j] = Hp[R - 1];
        my_f[j] = F;
        if constexpr (kEnds) {
          if (pk_max(best, thr) != thr) {  // rare: a cell of this column may be the optimum
            const uint32_t at = (my_col + j) << 16;
            if (pk_lo(best) > pk_lo(thr)) {
              const uint32_t v = best & 0xFFFFu;
              uint32_t row = 0;
#pragma unroll
              for (int k = R - 1; k >= 0; --k)
                if ((Hp[k] & 0xFFFFu) == v) row = k;
              const uint32_t key = at | (row0 + row);
              if (static_cast<int32_t>(v) > endsA || key < endA) {
                endsA = static_cast<int32_t>(v);
                endA = key;
              }
              thr = (thr & 0xFFFF0000u) | v;
            }
            if (pk_hi(best) > pk_hi(thr)) {
              const uint32_t v = best >> 16;
              uint32_t row = 0;
#pragma unroll
              for (int k = R - 1; k >= 0; --k)
                if ((Hp[k] >> 16) == v) row = k;
              const uint32_t key = at | (row0 + row);
              if (static_cast<int32_t>(v) > endsB || key < endB) {
                endsB = static_cast<int32_t>(v);
                endB = key;
              }
              thr = (thr & 0xFFFFu) | (v << 16);
            }
            if constexpr (MODE == kSw16End) g = pk_max(g, best);
          }
        }
      }
      hup_prev = h_in[C - 1];
      if constexpr (kEnds) {
        if (event && (ctl & kCtlLast)) {  // this lane's part of the task is done: fold its optimum into the task slot
          const int slot = static_cast<int>((ctl >> 24) & 7u);
          unsigned long long* e = s_end[warp][grp][slot];
          if (endsA > 0) atomicMax(e, (static_cast<unsigned long long>(endsA) << 32) | (0xFFFFFFFFu - endA));
          if (endsB > 0) atomicMax(e + 1, (static_cast<unsigned long long>(endsB) << 32) | (0xFFFFFFFFu - endB));
          if (feeder) {  // the group's last lane finishes the task last
#pragma unroll
            for (int h = 0; h < 2; ++h) {
              const uint32_t p = s_pair[own][grp][slot][h];
              if (p == kNoPair) continue;
              const unsigned long long x = e[h];
              const int32_t sc = static_cast<int32_t>(x >> 32);
              const uint32_t key = 0xFFFFFFFFu - static_cast<uint32_t>(x);
              if constexpr (MODE == kSw16End) {
                if (sc > thresh) {
                  prm.ovf_pairs[atomicAdd(prm.ovf_count, 1u)] = p;
                } else if (sc > 0) {  // a zero score keeps its cleared outputs
                  prm.scores[p] = sc;
                  prm.end_q[p] = static_cast<int32_t>(key & 0xFFFFu);
                  prm.end_t[p] = static_cast<int32_t>(key >> 16);
                }
              } else if (sc > 0) {
                prm.scores[p] = sc;
                prm.end_q[p] = static_cast<int32_t>(key & 0xFFFFu) - s_rev[warp][grp][slot][h].y;
                prm.end_t[p] = static_cast<int32_t>(key >> 16);
              }
            }
          }
        }
      } else if (event && (ctl & kCtlLast)) {  // this lane's part of the task is done: fold its maximum into the task slot
        const int slot = static_cast<int>((ctl >> 24) & 7u);
        atomicMax(&s_best[own][grp][slot][0], pk_lo(best));
        atomicMax(&s_best[own][grp][slot][1], pk_hi(best));
        best = 0;
        if (!TEAM && feeder) {  // the group's last lane finishes the task last: report both scores
          const int32_t bA = s_best[own][grp][slot][0], bB = s_best[own][grp][slot][1];
          const uint32_t pA = s_pair[own][grp][slot][0], pB = s_pair[own][grp][slot][1];
          if (pA != kNoPair) {
            if (bA > thresh) {
              prm.ovf_pairs[atomicAdd(prm.ovf_count, 1u)] = pA;
            } else {
              prm.scores[pA] = bA;
              if (prm.kernels) prm.kernels[pA] = 1u;
            }
          }
          if (pB != kNoPair) {
            if (bB > thresh) {
              prm.ovf_pairs[atomicAdd(prm.ovf_count, 1u)] = pB;
            } else {
              prm.scores[pB] = bB;
              if (prm.kernels) prm.kernels[pB] = 1u;
            }
          }
        }
      }
      // the bottom row of a pass that is not the last goes to the scratch line
      store_bnd<C>(feeder && (ctl & kCtlMore) != 0, bnd + my_col, my_h, my_f);
      my_col += C;
      if constexpr (TEAM) {
        if (feeder && (ctl & kCtlMore) && ((my_col & 15) == 0 || my_col == team_cols)) {
          __threadfence_block();  // the columns before their count
          s_prog[warp] = my_base + my_col;
        }
      }
      if (done) break;
      // the feeder's outgoing registers become lane 0's inputs for the next step; above the query's first row
      // H = 0 and the first-row F, else the previous pass's bottom row (which this lane stored)
      if (feeder) {
        my_ctl = n_ctl;
        my_rA = nA;
        my_rB = nB;
#pragma unroll
        for (int j = 0; j < C; ++j) {
          my_h[j] = 0;
          my_f[j] = F0;
        }
      }
      if constexpr (TEAM) {
        if (feeder && have && !gap && u_pass > 0) team_load();
      } else {
        load_bnd<C>(feeder && u_pass > 0, bnd + u_col, my_h, my_f);
      }
    }
    }  // have
    __syncthreads();
    if constexpr (TEAM) {
      if (threadIdx.x < 2) {  // both targets of the team's task
        const Sw16Slot sl = prm.slots[prm.warp_tasks[task.wt_begin].slot_begin + threadIdx.x];
        const int32_t b = s_best[0][0][0][threadIdx.x];
        if (sl.pair != kNoPair) {
          if (b > thresh || s_fail != 0) {
            prm.ovf_pairs[atomicAdd(prm.ovf_count, 1u)] = sl.pair;
          } else {
            prm.scores[sl.pair] = b;
            if (prm.kernels) prm.kernels[sl.pair] = 1u;
          }
        }
      }
      __syncthreads();  // before the next task's state is set up
    }
  }
}

}  // namespace st
