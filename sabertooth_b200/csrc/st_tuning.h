// Tile-class selection for the packed 16-bit kernel: lanes per alignment (G),
// query rows per lane (R) and columns per step (C).
//
// Batches: each query takes the class with the least estimated cost to the
// batch: the chip's time for its streamed cells (padded rows x padded columns x
// slots, from its own target lengths, over the class's measured rate; built-in
// B200 figures, replaced by st_autotune, 0 = class not considered), plus what its
// critical path exceeds the whole batch by.  A table entry per (query length,
// mean target length) bin, set by the caller, forces a class for that bin.
//
// Single alignments (the per-call path) take the class of the shortest
// critical path.
#pragma once
#include <algorithm>
#include <cstdint>

#ifdef __CUDACC__
#define TUNE_HD __host__ __device__
#else
#define TUNE_HD
#endif

constexpr int kTuneMBins = 10;  // query length: <=32, <=64, ..., <=8192, >8192
constexpr int kTuneNBins = 8;   // mean target length: <=64, <=128, ..., <=4096, >4096
constexpr int kMaxTileClasses = 32;

// The queries that the packed kernel stages: 22 int8 rows of the query padded to whole passes in shared memory, and a
// pass number that fits the eight bits it has in the kernel's control word (only <4,8> would need more, past 8,192 rows).
constexpr uint32_t kTuneStageBytes = 216 * 1024;
constexpr uint32_t kTuneMaxPasses = 256;

// The longest staged query, padded to whole passes of `rows` rows.
inline uint32_t tune_max_rows(uint32_t rows, uint32_t smem = kTuneStageBytes) {
  return std::min(std::min(smem, kTuneStageBytes) / 22 / rows, kTuneMaxPasses) * rows;
}

struct Tuning {
  int table[kTuneMBins][kTuneNBins];  // class index, -1 = rate model
  float rate[kMaxTileClasses];        // streamed cells per second / 1e12, per class; 0 = not used
};

int st_tuning_num_classes();
void st_tuning_class_shape(int c, int* G, int* R, int* C);
bool st_tuning_class_team(int c);
int st_tuning_class_warps(int c);

inline int tune_mbin(uint32_t m) {
  int b = 0;
  uint32_t lim = 32;
  while (b < kTuneMBins - 1 && m > lim) {
    ++b;
    lim <<= 1;
  }
  return b;
}

inline int tune_nbin(uint32_t n) {
  int b = 0;
  uint32_t lim = 64;
  while (b < kTuneNBins - 1 && n > lim) {
    ++b;
    lim <<= 1;
  }
  return b;
}

// Rates measured on B200 (148 SMs, 1965 MHz), streamed cells per second / 1e12,
// with every query of the PSSM workload (4,000 queries of 50-2,000 rows, 1.2 M
// pairs, targets of 160 residues on average) forced into one class.
inline float tuning_default_rate(int G, int R, int C, bool team) {
  if (C != 4) return 0.0f;
  static const struct {
    int G, R;
    float rate;
  } kRates[] = {
      {4, 8, 4.095f}, {8, 8, 4.718f}, {16, 8, 4.677f}, {32, 8, 4.762f},
      {4, 12, 3.985f}, {8, 12, 5.166f}, {16, 12, 5.248f}, {32, 12, 5.037f},
      {4, 16, 4.356f}, {8, 16, 5.331f}, {16, 16, 5.360f}, {32, 16, 5.190f},
      {4, 20, 4.543f}, {8, 20, 5.438f}, {16, 20, 5.442f}, {32, 20, 5.421f},
      {4, 24, 4.926f}, {8, 24, 5.766f}, {16, 24, 5.762f}, {32, 24, 5.444f},
      {4, 28, 5.305f}, {8, 28, 5.452f}, {16, 28, 5.471f}, {4, 32, 5.464f},
      {8, 32, 5.600f}, {16, 32, 5.615f}, {32, 32, 5.578f},
  };
  if (team) return 4.334f;
  for (const auto& r : kRates)
    if (r.G == G && r.R == R) return r.rate;
  return 0.0f;
}

inline void tuning_defaults(Tuning* t) {
  for (int i = 0; i < kTuneMBins; ++i)
    for (int j = 0; j < kTuneNBins; ++j) t->table[i][j] = -1;
  for (int c = 0; c < kMaxTileClasses; ++c) t->rate[c] = 0.0f;
  for (int c = 0; c < st_tuning_num_classes() && c < kMaxTileClasses; ++c) {
    int G, R, C;
    st_tuning_class_shape(c, &G, &R, &C);
    t->rate[c] = tuning_default_rate(G, R, C, st_tuning_class_team(c));
  }
}

// Columns that a team's task costs beside its longest target's: the lag of each further pass of a round, during
// which the CTA waits in part (a pass starts G + 5 steps after the one above it).
constexpr uint32_t kTeamLag = 5;
TUNE_HD inline uint32_t tune_team_cols(uint32_t G, uint32_t C, uint32_t P, uint32_t W) {
  return ((P < W ? P : W) - 1) * (G + kTeamLag) * C;
}

// Streamed cells of one query (m rows) in class c over its targets' lengths,
// sorted longest first: warp tasks of 64/G targets stream the longest one's
// length rounded up to 4 columns (at least C*G columns when the query takes
// several passes).
inline double tune_streamed(int c, uint32_t m, const uint32_t* tlen_desc, size_t n) {
  int G, R, C;
  st_tuning_class_shape(c, &G, &R, &C);
  const uint32_t rows = static_cast<uint32_t>(G * R);
  const uint32_t P = (m + rows - 1) / rows;
  if (P * rows > tune_max_rows(rows)) return 1e300;  // the class does not stage this query
  const uint32_t S = static_cast<uint32_t>(64 / G);
  uint32_t minc = 32;
  if (P > 1) minc = std::max<uint32_t>(minc, (static_cast<uint32_t>(C * G) + 15) & ~15u);
  double cols = 0;
  for (size_t w = 0; w < n; w += S) cols += std::max<uint32_t>(minc, (tlen_desc[w] + 3) & ~3u);
  if (st_tuning_class_team(c)) cols += static_cast<double>((n + S - 1) / S) * tune_team_cols(G, C, P, st_tuning_class_warps(c));
  return cols * S * P * rows;
}

// Critical path: the time of the wavefront that streams a query's longest target, alone on its scheduler, in
// picoseconds.  A step of a lone warp takes about 400 cycles (the shuffles, the profile loads, the dependent
// rows; 560 with 4 or 32 lanes) plus 11.8 for each of its R*C cell pairs; measured at 1,965 MHz on 4,000-column
// targets: <8,8> 771 cycles, <32,8> 938, <16,16> 1,182, <8,24> 1,541, <32,24> 1,570, <32,32> 1,932.  With a team of
// warps a pass starts G + 5 steps after the one above it, in rounds of `team` passes.
TUNE_HD inline double tune_crit_ps(uint32_t G, uint32_t R, uint32_t C, uint32_t P, uint32_t ncols, uint32_t team) {
  const double fixed = G == 8 || G == 16 || C == 2 ? 400.0 : 560.0;
  double steps = static_cast<double>(P) * (ncols / C);
  if (team > 1) {
    const uint32_t lag = G + kTeamLag, pass = ncols / C + G, round = pass > team * lag ? pass : team * lag;
    steps = static_cast<double>((P - 1) / team) * round + (P - 1) % team * lag + pass;
  }
  return (steps + G) * (fixed + 11.8 * (R * C)) * (1e6 / 1965.0);
}

// What a query costs the batch in a class: the chip's time for its cells, plus a part of what its critical path
// exceeds the whole batch by (batch_ps: the batch's time with every query in its cheapest class).  Large batches
// are all cell time and take the classes of few lanes, which pad least; in a small one the chip waits for the
// longest wavefront, so a query of many rows takes more lanes and fewer passes, or a team.  A path counts three
// times its lone length (a warp shares its scheduler with up to three others for most of its run), and its excess
// a tenth (the queries that exceed do so side by side).  Measured over factors 0-5 and weights 0.03-3: 100 PSSM
// queries x 300 targets 2.30 ms without the term, 1.44 with (1.5, 1), 1.10 with (3, 0.1); 600 queries 4.92, 4.83,
// 4.70 ms; 64 profiles x 1,000 samples 3.74, 2.42, 2.42 ms.
TUNE_HD inline double tune_objective(double est_ps, double crit_ps, double batch_ps) {
  const double over = 3.0 * crit_ps - batch_ps;
  return est_ps + (over > 0.0 ? 0.1 * over : 0.0);
}

// Warp tasks per unit of a CTA task: a CTA's warps; one on each scheduler where the batch has not two CTAs of them for
// every SM; fewer still (a power of two) while it would leave an SM without a unit, so that a small batch spreads over
// the chip.  Two thousand warp tasks in whole CTAs leave some SMs with two and others with one (4,000 spans 1.25 ms so,
// 1.09 by fours); one or two of eight warps at work share a scheduler while others idle (16 queries x 60 targets of 1,500 x
// 300 361 us by twos, 192 by eights).
TUNE_HD inline uint32_t tune_cta_unit(uint64_t wt_total, uint32_t sms, uint32_t W) {
  uint32_t u = W;
  if (u > 4 && static_cast<uint64_t>(u) * 2 * sms > wt_total) u = 4;
  while (u > 1 && static_cast<uint64_t>(u / 2) * sms >= wt_total) u >>= 1;
  return u;
}

// Whether every unit is a CTA task of its own: the whole batch is no more than the warps that are resident at once
// (two CTAs of eight warps on an SM, three of four).  A second unit in a task would be a second round of its warps
// while others have none; in larger batches it saves staging the query again (100 queries x 100 targets of 250 x 300 in
// <8,32>: 428 us with two units in most tasks, 233 with one; 600 queries x 300 of mixed lengths: 4.75 ms with one, 4.37).
TUNE_HD inline bool tune_cta_single(uint64_t wt_total, uint32_t sms, uint32_t W) {
  return wt_total <= static_cast<uint64_t>(sms) * (W < 8 ? 12 : 16);
}

// est[c] = the chip's time (ps) for the query in class c: streamed cells over the rate; a class without a rate
// counts 1e150 times its cells (taken only when no class with a rate stages the query), one that cannot stage it
// or is not in `allowed` 1e300.  Returns the least time over the classes with a rate (0: none).
inline double tuning_estimate(const Tuning* t, uint32_t m, const uint32_t* tlen_desc, size_t n, double* est,
                              uint32_t allowed) {
  double best = 0.0;
  for (int c = 0; c < st_tuning_num_classes(); ++c) {
    const double v = (allowed >> c & 1u) ? tune_streamed(c, m, tlen_desc, n) : 1e300;
    est[c] = v >= 1e300 ? 1e300 : (t->rate[c] > 0.0f ? v / t->rate[c] : v * 1e150);
    if (est[c] < 1e140 && (best == 0.0 || est[c] < best)) best = est[c];
  }
  return best;
}

// The class of one query of a batch (longest: its longest target); -1 when none stages it.
inline int tuning_pick_batch(const Tuning* t, uint32_t m, uint32_t longest, uint32_t mean_n, const double* est,
                             double batch_ps) {
  const int forced = t->table[tune_mbin(m)][tune_nbin(mean_n)];
  if (forced >= 0 && forced < st_tuning_num_classes() && est[forced] < 1e300) return forced;
  int best = -1;
  double bt = 1e300;
  for (int c = 0; c < st_tuning_num_classes(); ++c) {
    if (est[c] >= 1e300) continue;
    int G, R, C;
    st_tuning_class_shape(c, &G, &R, &C);
    const uint32_t rows = static_cast<uint32_t>(G * R), P = (m + rows - 1) / rows;
    const uint32_t minc = P > 1 ? std::max<uint32_t>(32, (static_cast<uint32_t>(C * G) + 15) & ~15u) : 32u;
    const double crit = tune_crit_ps(G, R, C, P, std::max<uint32_t>(minc, (longest + 3) & ~3u),
                                     st_tuning_class_team(c) ? st_tuning_class_warps(c) : 1);
    const double v = tune_objective(est[c], crit, batch_ps);
    if (v < bt) {
      bt = v;
      best = c;
    }
  }
  return best;
}

// The class in which a lone alignment of m rows and n columns is done first.
inline int tuning_pick_single(const Tuning*, uint32_t m, uint32_t n) {
  int best = 0;
  double bc = 1e301;
  for (int c = 0; c < st_tuning_num_classes(); ++c) {
    int G, R, C;
    st_tuning_class_shape(c, &G, &R, &C);
    const uint32_t rows = static_cast<uint32_t>(G * R), P = (m + rows - 1) / rows;
    if (P * rows > tune_max_rows(rows)) continue;  // the class does not stage this query
    uint32_t ncols = std::max<uint32_t>(32, (n + 3) & ~3u);
    if (P > 1) ncols = std::max<uint32_t>(ncols, (static_cast<uint32_t>(C * G) + 15) & ~15u);
    const double v = tune_crit_ps(G, R, C, P, ncols, st_tuning_class_team(c) ? st_tuning_class_warps(c) : 1);
    if (v < bc) {
      bc = v;
      best = c;
    }
  }
  return best;
}
