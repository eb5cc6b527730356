// Host rule that gives a GEMM its tile width (the columns of one scheduled tile).  Pure arithmetic, no CUDA
// calls, so that it can be checked without a GPU.
//
// The accumulator rows of a tile are fixed (128 per CTA); its columns may be any multiple of 32 up to 256.  A
// narrower tile reads more operand bytes per result, but lets a small problem reach more SMs, and lets a problem of
// a few waves fill its last wave.  The estimate counts SM cycles, with constants measured on a B200 at 1965 MHz:
//   a 64-deep k-block costs a CTA the longest of
//     the tensor work (546 cycles at 256 columns),
//     the issue loop of the producer (240 cycles and 45 for each TMA load: 64 to 160 columns take the same time), or of
//     the MMA warp, which comes to the same with two loads,
//     its share of what the L2 delivers to all active CTAs (10000 bytes a cycle, 95 to one CTA; half of that where K is not
//     a multiple of 64: 1152 x 2816 x 1000 14.8 us one-CTA, 13.2 in pairs.  What counts is rows that do not start on a
//     128-byte line, and K stands for the pitch of dense operands: an operand with a pitch of its own is judged by its K all
//     the same);
//   128 columns of epilogue cost 1700 cycles; the epilogue of one tile overlaps the k-blocks of the next, the last
//   one's is exposed; a CTA pair starts 2200 cycles later than a single CTA (cluster launch and barriers).
// A narrower width has to gain more than kMargin: estimates closer than that came out either way from one board to the
// next (512 x 8192 x 3584 in pairs: 224 columns 23.5 against 25.5 us on one, 28.1 against 24.8 us on another), and the wider tile reads less.
// Device times in us, 256 columns against the width taken: 128 x 8192 x 3584 one-CTA 23.1 -> 15.3 (128 columns),
// 384 x 3584 x 8192 47.5 -> 30.4 (128), 512 x 768 x 320 7.1 -> 5.5 (128), 2048 x 3584 x 8192 in pairs 111 -> 102 (224).
#pragma once
#include <cstdint>

namespace tcl {

constexpr int kMaxTileCols = 256;
constexpr int kTileColStep = 32;      // cta_group::2 MMAs take N in steps of 32
constexpr double kMargin = 0.10;

// Rows of one TMA box of B: a CTA's whole share of a tile, or for a gate|up tile narrower than the weight's blocks of
// 128 gate and 128 up rows the largest power of two in bn / 2, so that no box straddles two blocks.
inline int b_box_rows(int cta_group, int bn, bool gate_up) {
  if (!gate_up || bn == kMaxTileCols) return bn / cta_group;
  int box = 128;
  while ((bn / 2) % box != 0) box /= 2;
  return box;
}

// Estimated SM cycles of an m x n x k GEMM in tiles of (128 * cta_group) x bn on `ctas` CTAs.
inline double tile_cost(long long m, long long n, long long k, int cta_group, int ctas, int bn, bool gate_up, int split = 1) {
  const long long kb = ((k + 63) / 64 + split - 1) / split;
  const long long tiles = (m + 128 * cta_group - 1) / (128 * cta_group) * ((n + bn - 1) / bn);
  const int per = cta_group * split;
  const long long groups = ctas >= per ? ctas / per : 1;
  const long long waves = (tiles + groups - 1) / groups;
  const double active = static_cast<double>((tiles < groups ? tiles : groups) * per);
  // per CTA and k-block; rows of 128 bytes that do not start on a 128-byte line touch two
  const double bytes = (128.0 * 128.0 + 128.0 * bn / cta_group) * (k % 64 == 0 ? 1 : 2);
  double block = bn * (546.0 / 256.0);
  const double issue = 240.0 + 45.0 * (1 + bn / cta_group / b_box_rows(cta_group, bn, gate_up));
  if (block < issue) block = issue;
  if (block < bytes / 95.0) block = bytes / 95.0;
  if (block < bytes * active / 10000.0) block = bytes * active / 10000.0;
  const double main_loop = static_cast<double>(kb) * block;
  const double epilogue = 1700.0 * ((bn + 127) / 128);
  return static_cast<double>(waves) * (main_loop > epilogue ? main_loop : epilogue) + epilogue + (per > 1 ? 2200.0 : 0.0) +
         (split > 1 ? 1000.0 + (split - 1) * 512.0 * bn / split / 32.0 : 0.0);
}

// Columns per tile.
inline int pick_tile_cols(long long m, long long n, long long k, int cta_group, int ctas, bool gate_up) {
  int best = kMaxTileCols;
  double cost = tile_cost(m, n, k, cta_group, ctas, best, gate_up);
  for (int bn = kMaxTileCols - kTileColStep; bn >= kTileColStep; bn -= kTileColStep) {
    const double c = tile_cost(m, n, k, cta_group, ctas, bn, gate_up);
    if (c < cost * (1.0 - kMargin)) { best = bn; cost = c; }
  }
  return best;
}

// CTAs that share the k-blocks of a tile (one-CTA form), and that form's tile width with it: where the tiles do not fill
// the chip, a cluster per tile reads fewer operand bytes than narrower tiles would.  What it pays is a cluster launch,
// two cluster barriers and the exchange of (split - 1) / split of the fp32 accumulators (32 bytes a cycle).
// Without and with, us: 128 x 8192 x 3584 14.0 -> 11.6 (2 CTAs, 128 columns), 128 x 3584 x 8192 26.2 -> 13.3 (4, 128), 512 x 1024 x
// 8192 25.9 -> 13.5 (4, 128), 256 x 4096 x 4096 15.1 -> 12.4 (2, 128); not taken 256 x 4096 x 1024 6.8 against 7.9, 512 x 768 x 320 4.4 / 6.7.
struct SplitPick { int split, cols; };

// The width for a given split (2 or 4) and its estimate; no width (0) where the tiles do not fit the chip side by side or a
// CTA would get no k-block.
inline int pick_split_cols(long long m, long long n, long long k, int ctas, int split, double* cost) {
  int best = 0;
  for (int bn = kMaxTileCols; bn >= kTileColStep * split; bn -= kTileColStep * split) {
    const long long tiles = (m + 127) / 128 * ((n + bn - 1) / bn);
    if (tiles * split > ctas || (k + 63) / 64 < split) continue;
    const double c = tile_cost(m, n, k, 1, ctas, bn, false, split);
    if (best == 0 || c < *cost) { best = bn; *cost = c; }
  }
  return best;
}

inline SplitPick pick_split(long long m, long long n, long long k, int ctas, bool gate_up) {
  SplitPick best{1, pick_tile_cols(m, n, k, 1, ctas, gate_up)};
  if (gate_up) return best;
  double cost = tile_cost(m, n, k, 1, ctas, best.cols, false) * (1.0 - kMargin);
  for (int split = 2; split <= 4; split *= 2) {
    if ((k + 63) / 64 < 4 * split) continue;
    // fours do not fill a GPC of the chip whose SMs are no multiple of four: leave some room
    const int room = split == 4 ? ctas - ctas / 8 : ctas;
    double c = 0.0;
    const int bn = pick_split_cols(m, n, k, room, split, &c);
    if (bn != 0 && c < cost) { cost = c; best = {split, bn}; }
  }
  return best;
}

// One CTA or a pair per tile, for rows that are a multiple of 128 (the pair's last tile may be half empty).  The pair
// reads a third less from the L2; the single CTA starts earlier.  One-CTA against pair, us: 512 x 768 x 320 5.5 / 6.6,
// 256 x 4096 x 4096 16.7 / 17.6, 512 x 8192 x 1024 11.2 / 12.2, 512 x 8192 x 3584 28.0 / 24.8, 4992 x 4096 x 4096 147 / 142.
inline int pick_cta_group(long long m, long long n, long long k, int ctas) {
  const SplitPick s = pick_split(m, n, k, ctas, false);
  const double one = tile_cost(m, n, k, 1, ctas, s.cols, false, s.split);
  const double pair = tile_cost(m, n, k, 2, ctas, pick_tile_cols(m, n, k, 2, ctas, false), false);
  return one < pair ? 1 : 2;
}

// Two adjacent 256-column tiles per work item (pair form only).  Large problems are bound by power: the tensor pipe is
// active 92 % of the cycles, at whatever clock the power allows, so bytes not moved are time.  256 x 512 reads a quarter
// less from the L2 than 256 x 256, but both accumulator buffers belong to one item and its epilogue is hidden only by
// the skew at its ends.  Sustained, us, 256 against 512 columns: 8192^3 885 -> 843, 16384 x 7168 x 8192 1581 -> 1465,
// 32768 x 28672 x 8192 13.3 -> 12.5 ms, 16384 x 8192 x 3584 758 -> 738, but K = 1024 (32768 x 8192) 453 -> 470, and with 2.2
// waves of items (4992 x 4096 x 4096) 141 -> 145.  Around the two lines, each width run alone until its clock settled: 16384 x
// 8192 with K = 1536 320 -> 330, 2048 421 -> 422, 2560 520 -> 516, 3072 619 -> 611, 3584 718 -> 709; with K = 4096 and 3.5 waves
// (4096 x 8192) 208 -> 208, 4.3 waves 263 -> 267, 6.9 waves 413 -> 406; with K = 8192 and 2.6 waves 333 -> 325, 3.5 waves 419 -> 411,
// 4.3 waves 533 -> 517.  The lines lie inside the band where the two differ by under 3 %.
constexpr int kWideMinK = 3072;
constexpr int kWideMinWaves = 4;
// Raster group of wide tiles, in tile rows: 16 x 256 rows by 4.6 x 512 columns is what 74 pairs work on at a time, nearer
// to a square than with 8 rows (8192^3 846 -> 830 us, 16384 x 7168 x 8192 1515 -> 1458 us).
constexpr int kWideGroupM = 16;

inline bool pick_wide(long long m, long long n, long long k, int ctas) {
  const long long pairs = ctas / 2;
  return k >= kWideMinK && pairs > 0 && (m + 255) / 256 * ((n + 511) / 512) >= kWideMinWaves * pairs;
}

// Columns per work item: a tile's, or 512 for two of 256.
inline int pick_cols(long long m, long long n, long long k, int cta_group, int ctas, bool gate_up) {
  const int bn = pick_tile_cols(m, n, k, cta_group, ctas, gate_up);
  return cta_group == 2 && bn == kMaxTileCols && pick_wide(m, n, k, ctas) ? 2 * kMaxTileCols : bn;
}

}  // namespace tcl
