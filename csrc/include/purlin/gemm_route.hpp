// Which kernel a GEMM takes and how it is cut: rules on sizes and on what the device holds, host arithmetic alone, so that they
// are tested without a GPU (csrc/tests/cpu_unit_test.cpp). The kernels: the tiles of gemm_sm100.cu (plain), gemm_skinny.cuh (few
// rows), gemm_ragged.cuh (any number of rows).
#pragma once
#include <algorithm>
#include <cmath>
#include <cstddef>
#include <cstdint>

namespace purlin {

namespace skinny {
constexpr int kRows = 128, kK = 64;            // rows of W per tile, k per stage (128-byte swizzled rows)
constexpr int kWBytes = kRows * kK * 2;
constexpr int kMaxStages = 8;
constexpr int kMaxTokens = 256;                // columns of one pass
constexpr int kBarrierBytes = 256;
constexpr int kMaxSplit = 8;
}  // namespace skinny

namespace ragged {
constexpr int kBM = 128, kBK = 64, kMaxCols = 256;
constexpr int kABytes = kBM * kBK * 2;
constexpr int kAccRows = 256;                   // rows of W per accumulator of a pair; a tile has one or two of them
constexpr int kMaxStages = 8, kRingBytes = 192 * 1024;
constexpr int kXBox = 32;                       // rows of one X load
constexpr int kNarrowCols = 64;                 // columns of a tile that leave room for a fifth stage
}  // namespace ragged

namespace route {

// Whether a launch is better placed on an empty GPU. Between half as many CTAs as SMs and six sevenths of them, a kernel that is
// set up early takes the SMs its predecessor leaves free and then some of those it gives back, so neighbouring SMs that share
// their path to L2 are both busy, where a launch on its own would have spread out. Where the main loop is short, the microsecond
// that the overlap saves is more than that costs; from 28 k-blocks on it is not. Apart / overlapped, us: 6148 x 448 x 7000 SwiGLU
// (98 CTAs) 64.5 / 72.6, 108 x 12672 x 2584 (99) 21.4 / 24.9, 7822 x 384 x 5064 (124) 44.6 / 49.6. Of 1074 shapes on these tiles
// the overlap slows 32 by more than 5 %; with this rule two, and two that gained more than 3 % lose it.
inline bool betterApart(long ctas, int K, int sms) { return ctas * 2 > sms && ctas * 7 < sms * 6 && K >= 28 * ragged::kBK; }

// Which GEMMs the few-rows kernel takes, each line with one B200's times in us, it / the other tiles. Few rows of W (a router)
// with a long k: 4096 x 32 x 7168 11 / 75; with a short k the sum over the partial tiles costs more than it saves (1656 x 208
// x 112 14.4 / 12.2 a call).
inline bool fewWeightRows(int M, int N, int K, bool swiglu) { return !swiglu && M > skinny::kMaxTokens / 2 && N <= skinny::kMaxTokens && K >= 2048; }
inline bool useSkinny(int M, int N, int K, bool swiglu) {
  if (fewWeightRows(M, N, K, swiglu)) return true;
  // always up to 32 rows, up to 64 once k is long enough to be split: 64 x 4096 x 1024 7.9 / 8.3, 54 x 7648 x 1336 SwiGLU 14.3 / 17.2;
  // but 64 x 104 x 144 5.6 / 3.8, 64 x 22968 x 72 9.2 / 6.4. Above, what the others would take decides (kernelOf).
  return M <= 64 && (M <= 32 || K >= (N <= 8192 ? 512 : 1024));
}
// Parts that the few-rows kernel cuts k into: while the CTAs have a place on the GPU at the same time and a part keeps at least four
// k-blocks; eight where many tiles are split four ways (64 x 7744 x 1160, 61 tiles: 12.0 us whole, 10.6 in two parts, 13.0 in four).
// Measured, 1 x 8192 x 3584: one CTA per tile 20.1 us, two 14.4, four 14.2, eight 18.2; 64 x 8192 x 28672: 142.6 / 87.4 / 79.1 /
// 90.5 us. More CTAs than places cost a second wave: 64 x 11232 x 1952 SwiGLU (88 tiles, 296 places) 16.6 / 14.7 / 26.7,
// 192 x 5824 x 1280 (46 tiles, 148 places) 17.0 / 13.1 / 23.9. At most 15 clusters of eight fit on the GPU at once, so eight
// are used for no more tiles than that.
inline int skinnySplit(long tiles, int kBlocks, long slots) {
  int split = 1;
  while (split < (tiles <= 15 ? skinny::kMaxSplit : 4) && tiles * split * 2 <= slots && kBlocks >= (split > 1 && tiles > 24 ? 16 : 8) * split) split *= 2;
  return split;
}

// CTAs that share the columns of a tile, where its k parts leave SMs without one: a k-block takes 450 cycles and 3.5 per column, and the
// few rows of W that they all read come from L2 (fifteen clusters of eight fit on the GPU). In a graph, us, one CTA for all columns /
// shared: 128 x 32 x 7168 9.8 / 7.5, 128 x 256 x 4096 10.9 / 7.1, 200 x 512 x 7168 17.4 / 12.0, 300 x 256 x 7168 16.5 / 9.6, 128 x 2048 x 4096
// 13.8 / 11.4, 50 x 600 x 1000 6.7 / 5.4. More than half the SMs only for parts of six k-blocks: 40 x 2048 x 1024 5.7 / 6.3.
inline int skinnyGroups(int columns, long tiles, int split, int kBlocks, int sms) {
  const long ctas = std::max(tiles * split, 1l), places = kBlocks >= 6 * split ? sms : sms / 2;
  const long room = split == skinny::kMaxSplit ? 15 / std::max(tiles, 1l) : places / ctas;
  return int(std::max(std::min(long(columns + 31) / 32, room), 1l));
}

struct SkinnyCut {
  int tokenBox, passTokens, split, columnGroups, stages, stageBytes, tmemCols;
  int ahead;       // k-blocks of W that a CTA asks into L2 before the kernel before it has ended
  bool apart;      // not set up while the kernel before it runs
};
// M columns of the MMA (rows of X), N rows of W per expert. likelyRows > 0: grouped, rows that an expert is expected to have.
inline SkinnyCut skinnyCut(int M, int N, int K, int experts, int likelyRows, int sms) {
  SkinnyCut c{};
  auto up = [](int v, int to) { return (v + to - 1) / to * to; };
  // one pass has to hold a group's rows (a second pass reads W again): a group of average size has twice the room
  const int room = int(std::min<int64_t>(likelyRows > 0 ? 2 * int64_t(likelyRows) + 16 : M, M));
  c.tokenBox = room <= 16 ? 16 : 32;
  c.passTokens = std::min(up(std::min(room, skinny::kMaxTokens), c.tokenBox), skinny::kMaxTokens);
  const int tiles = (N + skinny::kRows - 1) / skinny::kRows, kBlocks = (K + skinny::kK - 1) / skinny::kK;
  c.split = skinnySplit(long(tiles) * experts, kBlocks, long(sms) * (c.passTokens <= 128 ? 2 : 1));
  c.columnGroups = 1;
  if (!likelyRows && M <= c.passTokens) {
    c.columnGroups = skinnyGroups(M, tiles, c.split, kBlocks, sms);
    c.passTokens = up((M + c.columnGroups - 1) / c.columnGroups, c.tokenBox);
    c.columnGroups = (M + c.passTokens - 1) / c.passTokens;      // (160 columns for four: 64 each, and nothing for the fourth)
  }
  // up to 128 columns two CTAs share an SM (128 columns: 3 stages of 32 KiB each)
  c.stageBytes = skinny::kWBytes + c.passTokens * skinny::kK * 2;
  const int perSm = c.passTokens <= 128 ? 2 : 1;
  const int budget = (perSm == 2 ? 113 : 227) * 1024 - 1024 - skinny::kBarrierBytes;
  c.stages = std::min(budget / c.stageBytes, skinny::kMaxStages);
  for (c.tmemCols = 32; c.tmemCols < c.passTokens; c.tmemCols *= 2) {}
  // Between half as many CTAs as SMs and as many, they are better placed on an empty GPU, one to an SM: set up early they pile
  // up two to an SM where the kernel before left room (97-token MLP block 5824 x 1888, 120 CTAs: 40.7 us apart, 42.5 overlapped).
  const long ctas = long(tiles) * c.split * experts * c.columnGroups;
  // With shared columns the tiles are small and the launch is the larger part: 200 x 2048 x 4096 15.1 us apart, 13.7 overlapped.
  c.apart = ctas * 2 > sms && ctas < sms && c.columnGroups == 1;
  // Grouped, nobody knows yet which experts have rows: a lap of every idle expert's ring was up to four times the bytes that the call
  // needs (MoE block 7168 / 2048 with / without it, us, one token: top-1 of 32 100.4 / 84.0, top-1 of 64 114.7 / 92.2,
  // top-8 of 64 215 / 184; two tokens, top-8 of 64 306 / 279).
  c.ahead = c.apart || likelyRows ? 0 : c.stages;
  return c;
}

constexpr int kFewGroupRows = 12;
constexpr int kMaxParts = 4;            // pairs of a cluster (eight CTAs, the largest portable cluster)
// stages of a ring for `accs` accumulators and `cols` columns per tile
inline int raggedStages(int accs, int cols, uint32_t& stageBytes) {
  stageBytes = uint32_t(accs * ragged::kABytes + (cols / 2 + ragged::kXBox - 1) / ragged::kXBox * ragged::kXBox * ragged::kBK * 2);
  return std::min(int(ragged::kRingBytes / stageBytes), ragged::kMaxStages);
}

// How the ragged kernel cuts a GEMM: one or two accumulators per tile, the number of column tiles, and how many pairs share a tile's k
// range, whichever has the least expected time. The cycles are a model, its constants fitted to about 700 shapes on one B200:
//   a k-block of a tile of two accumulators takes the tensor pipe 4 cycles a column, and its operands come at 44 bytes a cycle and SM;
//   of one accumulator 500 and 2.1 a column (the round trips of its loads); rows of K that begin off a cache line 12 % more;
//   drain: what a tile's epilogue exposes; behind the last one its stores remain;
//   a cluster of several pairs is placed later than a pair (3500 cycles a pair) and exchanges partial tiles at 12 bytes a cycle;
//   the weights come through HBM once.
// What it buys, us, one B200, before / now: 2048 x 14336 x 8192 SwiGLU 371 / 325 (ten column tiles, where eight left a fourth wave of two
// tiles), 1000 x 14336 x 8192 SwiGLU 205 / 168, 1000 x 8192 x 7168 97 / 85, 384 x 14336 x 8192 SwiGLU 121 / 78, 700 x 8192 x 28672 428 / 250;
// with k split over two pairs 512 x 8192 x 28672 297 / 174, 384 x 8192 x 28672 224 / 142, 200 x 14336 x 8192 SwiGLU 70 / 58.
struct RaggedPlan { int tileAccs = 2, colTiles = 1, tiles = 1, parts = 1; double cycles = 0; };
inline RaggedPlan raggedPlan(int M, int N, int K, bool swiglu, const int (&clusters)[3]) {
  const int kBlocks = (K + ragged::kBK - 1) / ragged::kBK, units = (M + 31) / 32, fewest = (units + 7) / 8;
  const double unaligned = K % ragged::kBK ? 1.12 : 1.;                 // rows of K that do not begin on a cache line
  auto cyclesOf = [&](int accs, double cols, int64_t tiles, int parts) {
    auto perBlock = [&](int a) {
      if (a == 1) return (500 + 2.1 * cols) * unaligned;
      return std::max(4 * cols, (2 * ragged::kABytes + cols * 64) / 44 * unaligned);
    };
    auto drain = [&](int a) { return 1200. + a * cols * (swiglu ? 8. : 3.); };
    const int places = clusters[parts / 2];
    const int64_t full = tiles / places, rest = tiles % places;
    const double whole = (kBlocks + parts - 1) / parts * perBlock(accs) + drain(accs) + (parts > 1 ? 3500. * parts + accs * cols * 512. * (parts - 1) / parts / 12 : 0.);
    const double tail = rest == 0 ? 0. : parts == 1 && accs == 2 && 2 * rest <= places ? kBlocks * perBlock(1) + drain(1) : whole;
    // the weights once through HBM, at least
    return std::max(double(full) * whole + tail, (2. * N * K + 2. * M * K) / 3300. * unaligned) + 4500. + accs * cols * 8.;
  };
  RaggedPlan best;
  double bestKey = 0;
  for (int accs = 1; accs <= 2; ++accs) {
    // the fewest column tiles, one and two more, tiles of at most 7 to 4 units (of 32 rows), and the numbers that just fill one to three
    // waves more than the fewest need
    const int64_t wTiles = (N + accs * ragged::kAccRows - 1) / (accs * ragged::kAccRows), waves = fewest * wTiles / clusters[0];
    for (int c = 0; c < 10; ++c) {
      const int64_t want = c < 3 ? fewest + c : c < 7 ? (units + 9 - c) / (10 - c) : (waves + c - 6) * clusters[0] / wTiles;
      if (want < fewest || want > units || want > 2 * fewest + 2) continue;
      const int n = int(want);
      const int64_t tiles = n * wTiles;
      const double average = 32. * units / n, widest = (units + n - 1) / n * 32;
      for (int parts = 1; parts <= kMaxParts; parts *= 2) {
        if (!clusters[parts / 2] || kBlocks < 8 * parts || (parts > 1 && tiles > clusters[parts / 2])) break;
        // Among cuts: a pair with few tiles has the widest among them, and narrow tiles move more bytes per operation, which costs power
        // (2072 x 4800 x 5016 SwiGLU: 11 tiles of 192 88.7 us, 14 of 128 and 160 97.2). Between kernels the plain number of cycles chooses better
        // (one factor for all K off a cache line, 914 shapes: 2.2 % above the best kernel of each; with this factor 2.5 %).
        const double key = cyclesOf(accs, average + (widest - average) * clusters[0] / std::max<int64_t>(tiles, clusters[0]), tiles, parts) * (0.95 + 12.8 / average);
        if (bestKey == 0 || key < bestKey) {
          bestKey = key;
          best = RaggedPlan{accs, n, int(std::min<int64_t>(tiles, INT32_MAX / 4)), parts, cyclesOf(accs, average, tiles, parts)};
        }
      }
    }
  }
  return best;
}

struct RaggedCut {
  int tileAccs, colTiles, maxCols, parts, stages, narrowStages;
  uint32_t stageBytes, narrowStageBytes;
  int grid;        // CTAs
  bool apart;      // not set up while the kernel before it runs
};
// plan: of a GEMM of M rows; null: grouped, the tiles of each expert are known on the device. pairs: that the device holds.
inline RaggedCut raggedCut(int M, int K, const RaggedPlan* plan, int pairs, int sms) {
  RaggedCut c{};
  c.tileAccs = 2; c.colTiles = 1; c.parts = 1;
  c.maxCols = ragged::kMaxCols;
  int items = INT32_MAX;
  if (plan) {
    c.tileAccs = plan->tileAccs; c.colTiles = plan->colTiles; c.parts = plan->parts;
    c.maxCols = ((M + 31) / 32 + plan->colTiles - 1) / plan->colTiles * 32;
    items = plan->parts > 1 ? plan->tiles : plan->tileAccs * plan->tiles;      // (the tiles of a small last wave are issued as halves)
  }
  c.stages = raggedStages(c.tileAccs, c.maxCols, c.stageBytes);
  // (grouped, the kernel decides between wide and narrow tiles: it knows the counts)
  c.narrowStages = raggedStages(c.tileAccs, std::min(c.maxCols, ragged::kNarrowCols), c.narrowStageBytes);
  c.grid = (c.parts > 1 ? items : std::min(pairs, items)) * 2 * c.parts;
  // Fewer tiles than pairs: the pairs without one leave at once. Tiles of one accumulator are better overlapped all the same (14 shapes of 38
  // to 63 tiles: apart 1.02 to 1.10 of the time overlapped; of two accumulators 0.91 to 1.05, 0.995 on average).
  c.apart = c.parts > 1 ? betterApart(c.grid, K, sms) : plan && plan->tileAccs == 2 && betterApart(2l * std::min(pairs, plan->tiles), K, sms);
  return c;
}

struct PlainTiles { int tilesM, tilesN, bn, ctas, accs; };
// The plain tiles of this file on the same scale.
inline double plainCycles(const PlainTiles& t, int M, int N, int K, bool swiglu, int sms) {
  const double tiles = double(t.tilesM) * t.tilesN, places = t.ctas == 2 ? sms / 2 : sms;
  const double block = t.accs == 2 ? std::max(4. * t.bn, 900.) : std::max({2. * t.bn + 184., (ragged::kABytes + t.bn / t.ctas * 128) / 58., 700.});
  const double drain = t.accs == 2 ? (swiglu ? 9000. : 6000.) * t.bn / 256 : 0.;
  const double waves = std::ceil(tiles / places);
  // rows of K that do not begin on a cache line; or not even on a sector of 32 bytes, which costs least where W has few rows to load
  const double unaligned = K % ragged::kBK == 0 ? 1. : K % 16 == 0 ? 1.1 : N > 128 ? 1.55 : 1.15;
  return std::max(waves * ((K + ragged::kBK - 1) / ragged::kBK * block * unaligned + drain) + 3000., (2. * N * K + 2. * M * K) / 3300. * unaligned);
}

// ... and the few-rows kernel: its CTAs' round trips (per k-block 450 cycles and 3.5 per column, measured with L2-sized weights) and what
// each CTA adds at its end, which grows with the rows (the partial tiles through distributed shared memory), or the weights. CTAs beyond
// those that the device holds are a second wave: at one CTA an SM 33 clusters of four and 15 of eight fit (151 x 4568 x 2256, 36
// clusters of four: 25 us, the ragged kernel 16).
inline double skinnyCycles(int M, int N, int K, bool swiglu, int sms) {
  if (M > skinny::kMaxTokens || N > 16384) return 1e30;
  const long tiles = (N + skinny::kRows - 1) / skinny::kRows;
  const SkinnyCut c = skinnyCut(M, N, K, 1, 0, sms);
  const int kBlocks = (K + skinny::kK - 1) / skinny::kK, width = (M + c.columnGroups - 1) / c.columnGroups;
  const long places = long(c.split == 8 ? std::min(sms, 120) : c.split == 4 ? std::min(sms, 132) : sms) * (M <= 128 ? 2 : 1);
  const double waves = std::ceil(double(tiles * c.split) / places), block = (450. + 3.5 * ((width + 31) / 32 * 32)) * (tiles * c.split > sms ? 1.3 : 1.);
  const double end = (swiglu ? 105. : 45.) * M;
  return std::max(waves * (double(kBlocks) / c.split * block + end), 1.15 * (2. * N * K + 2. * M * K) / 3300. + end) + 7000.;
}

// The least expected time. The ragged kernel was 3 % ahead of the plain tiles at 4096 x 8192 x 7168 (326 / 351 us) and 8192 x 2048 x 1024
// (28.8 / 30.7), behind at 2048 x 4096 x 512 (13.8 / 12.1) and 1000 x 4096 x 4096 (36 / 33, one wave of narrower tiles); the few-rows
// kernel ahead at 128 x 8192 x 8192 (33.6, ragged 37.5, plain 42.2), behind at 128 x 8192 x 2048 (18.2, plain 13.9) and 160 x 8192 x
// 8192 (38.6, ragged 36.6). The models are not good to a few per cent, and for tiles of one accumulator the ragged one is more hopeful than
// the plain one (by 8 % in the medians of measured over expected), so such a cut has to be expected ahead by 5 %. Of 914 random shapes, every
// kernel timed on each, the choice then takes 1.6 % longer than the best kernel on average, and 14 are more than 3 % slower than by the
// tile counts that decided before there was a model. Without that margin, with one factor for all K off a cache line and without the second
// waves of the few-rows kernel it was 2.4 % and 41 (2006 x 64 x 1320 plain 12.4 us, ragged 16.5; 151 x 4568 x 2256 ragged 16, few rows 25).
enum { kPlain = 0, kSkinny = 1, kRagged = 2 };
inline int kernelOf(double plain, double skinny, double ragged, int tileAccs) {
  if (tileAccs == 1) ragged *= 1.05;
  return skinny < std::min(plain, ragged) ? kSkinny : ragged < plain ? kRagged : kPlain;
}

}  // namespace route
}  // namespace purlin
