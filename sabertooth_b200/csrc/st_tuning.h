// Tile-class selection for the packed 16-bit kernel: lanes per alignment (G),
// query rows per lane (R) and columns per step (C).
//
// Batches: each query's classes are weighed by the chip's time for its streamed
// cells (padded rows x padded columns x slots, from its own target lengths, over
// the class's measured rate; built-in B200 figures, replaced by st_autotune, 0 =
// class not considered) and by their critical paths.  A table entry per (query
// length, mean target length) bin, set by the caller, forces a class for that bin.
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

// What a class costs a query of a batch: the chip's time for its cells, the length of its critical path, and the turns
// its warp tasks take of an SM's four schedulers.  A large batch is all cell time and takes the classes of few lanes,
// which pad least; a small one waits for its longest wavefront, so a query of many rows takes more lanes and fewer
// passes, or a team.  How the two are weighed depends on how alike the paths are (tune_alike).
struct TuneCost {
  double est;     // the streamed cells over the rate; >= 1e140: a class without a rate, 1e300: it does not stage the query
  double ps;      // the same with what a small batch pays beside
  double path;
  double rounds;
};

// nw: warp tasks, in CTAs of W warps.  A wavefront starts and ends with G - 1 steps of idle lanes, once for the warp
// tasks that a warp streams one after the other: each in a batch that fits the chip (batch_ps, its cell time in the
// cheapest classes, below the three and a half paths of a full scheduler), up to sixteen in a large one.  And a CTA holds
// one query, so many queries of a few warp tasks each take the places of the CTAs that fit the chip, two on an SM or
// three of four warps or eight rows a lane.
TUNE_HD inline TuneCost tune_cost(uint32_t G, uint32_t R, uint32_t C, uint32_t W, bool team, uint32_t P,
                                  uint32_t longest_cols, uint32_t nw, double est_ps, double rate, double batch_ps,
                                  uint32_t sms) {
  TuneCost r{est_ps, est_ps, tune_crit_ps(G, R, C, P, longest_cols, team ? W : 1), 0.0};
  r.rounds = team ? nw * (W / 4) : nw / W * (W / 4) + (nw % W + 3) / 4;
  if (est_ps < 1e140) {
    const double streamed = batch_ps / (3.5 * r.path);
    const double ramp = 64.0 * R * C * (G - 1) * nw / rate;  // a step is 64 R C cells of a warp
    r.ps += ramp / (streamed < 1.0 ? 1.0 : (streamed > 16.0 ? 16.0 : streamed));
    const double place = r.path / ((W < 8 || R == 8 ? 3.0 : 2.0) * sms) * (team ? nw : 1u);
    if ((team || nw < W) && place > r.ps) r.ps = place;
  }
  return r;
}

// Paths of mixed lengths: each query is weighed by itself, the time of its cells and a tenth of what its path exceeds the
// whole batch by.  A path counts three times its lone length (a warp shares its scheduler with up to three others for
// most of its run), and a tenth because the queries that exceed do so side by side.  100 PSSM queries x 300 targets 2.30
// ms without the second term, 1.10 with it; 600 queries 4.92 and 4.70 ms.
TUNE_HD inline bool tune_waits(double path, double batch_ps) { return 3.0 * path > batch_ps; }
TUNE_HD inline double tune_weighed(const TuneCost& c, double batch_ps) {
  return c.est + (tune_waits(c.path, batch_ps) ? 0.1 * (3.0 * c.path - batch_ps) : 0.0);
}

// Paths much alike, the longest (of the queries in their cheapest classes) within a quarter of the mean, and most of
// them waited for: that would count one path once for each query.  The batch has one limit for the paths instead: each query
// takes the class of least time whose path is within it (the shortest path where none is), and the limit is the one of
// the least estimate of the batch's time, from the sums of its queries' times and rounds and its longest path.  That
// wavefront shares its scheduler with as many others as there are rounds, up to two more, and a third of what is the
// shorter of its time and the cells' comes on top.  Microseconds with each query by itself / with a limit: 64 queries x
// 60 targets of 250 x 300 132 / 101, 100 x 100 303 / 255, 300 x 50 of 100 x 160 162 / 116, 64 x 60 of 600 x 300 274 / 230.
// With mixed lengths the limit lost as much as it won: 16 x 300 766 / 717, 100 x 300 1,375 / 1,740.
TUNE_HD inline bool tune_alike(double longest_path, double path_sum, uint64_t n, uint64_t n_wait) {
  return 2 * n_wait > n && longest_path * n <= 1.25 * path_sum;
}
TUNE_HD inline double tune_batch_time(double cells_ps, double path_ps, double rounds, uint32_t sms) {
  const double load = rounds / sms;
  const double path = path_ps * (load < 1.0 ? 1.0 : (load > 3.0 ? 3.0 : load));
  return cells_ps > path ? cells_ps + path / 3.0 : path + cells_ps / 3.0;
}

// The limits that are compared: the longest path of the queries in their cheapest classes, and down from it in steps of
// a tenth.
constexpr int kTuneLimits = 32;
TUNE_HD inline double tune_limit(double longest, int i) {
  for (; i > 0; --i) longest *= 0.9;
  return longest;
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

// The class that the table forces on a query, -1: none, or it does not stage the query.
inline int tuning_forced(const Tuning* t, uint32_t m, uint32_t mean_n, const double* est) {
  const int forced = t->table[tune_mbin(m)][tune_nbin(mean_n)];
  return forced >= 0 && forced < st_tuning_num_classes() && est[forced] < 1e300 ? forced : -1;
}

// Every class's cost for a query of m rows, n targets of which the longest has `longest` residues, from its estimates.
inline void tuning_costs(const Tuning* t, uint32_t m, uint32_t longest, size_t n, const double* est, double batch_ps,
                         uint32_t sms, TuneCost* cost) {
  for (int c = 0; c < st_tuning_num_classes(); ++c) {
    int G, R, C;
    st_tuning_class_shape(c, &G, &R, &C);
    const uint32_t rows = static_cast<uint32_t>(G * R), P = (m + rows - 1) / rows, S = static_cast<uint32_t>(64 / G);
    const uint32_t minc = P > 1 ? std::max<uint32_t>(32, (static_cast<uint32_t>(C * G) + 15) & ~15u) : 32u;
    cost[c] = tune_cost(G, R, C, st_tuning_class_warps(c), st_tuning_class_team(c), P,
                        std::max<uint32_t>(minc, (longest + 3) & ~3u), static_cast<uint32_t>((n + S - 1) / S), est[c],
                        t->rate[c], batch_ps, sms);
  }
}

// The classes that some limit picks for a query, shortest path first and each cheaper than those before it: under a limit
// the query takes the last whose path is within it, or the first.  Without a class that has a rate the cheapest that
// stages the query alone.  Returns their number (0: none stages it).
inline int tuning_front(const TuneCost* cost, uint8_t* front) {
  uint8_t order[kMaxTileClasses];  // the classes with a rate by path, then time
  int m = 0, unrated = -1;
  for (int c = 0; c < st_tuning_num_classes(); ++c) {
    if (cost[c].ps >= 1e140) {
      if (cost[c].ps < 1e300 && (unrated < 0 || cost[c].ps < cost[unrated].ps)) unrated = c;
      continue;
    }
    int i = m++;
    for (; i > 0; --i) {
      const TuneCost& o = cost[order[i - 1]];
      if (o.path < cost[c].path || (o.path == cost[c].path && o.ps <= cost[c].ps)) break;
      order[i] = order[i - 1];
    }
    order[i] = static_cast<uint8_t>(c);
  }
  int n = 0;
  for (int i = 0; i < m; ++i)
    if (n == 0 || cost[order[i]].ps < cost[front[n - 1]].ps) front[n++] = order[i];
  if (n == 0 && unrated >= 0) front[n++] = static_cast<uint8_t>(unrated);
  return n;
}

// The class of a query by its own weight (tune_weighed); -1 when none stages it.
inline int tuning_weighed(const TuneCost* cost, double batch_ps) {
  int best = -1;
  for (int c = 0; c < st_tuning_num_classes(); ++c)
    if (cost[c].est < 1e300 && (best < 0 || tune_weighed(cost[c], batch_ps) < tune_weighed(cost[best], batch_ps))) best = c;
  return best;
}

// Its place among them under a limit.
inline int tuning_under(const TuneCost* cost, const uint8_t* front, int n, double limit) {
  while (n > 1 && cost[front[n - 1]].path > limit) --n;
  return n - 1;
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
