// GEMM for any number of activation rows, plain or per expert: C[T, N] = X[T, K] * W[N, K]^T on CTA pairs.
//
// What bounds it is the tensor pipe, and the loss it removes is padding: the rows of X (a prompt chunk, the rows of an
// expert) are no multiple of a 256- or 512-row tile. So W fills the rows of the MMA (its row count is a multiple of the
// tile in practice) and the rows of X are the columns, whose number may be any multiple of 32: T rows are shared out over as many
// column tiles as leave the pairs least idle (rows of 1030 in five tiles of 192 to 224 and not four of 256 and one of 32: the loads
// of W make a narrow tile dear).
//   * a tile is 512 rows of W (two accumulators of a CTA pair, 256 rows each) x up to 256 rows of X; the two accumulators
//     share the X operand, and their MMAs alternate: an MMA waits for the one before into the same columns (174 cycles instead of
//     128, measured). Where there are few tiles a tile is 256 rows of W. A last wave that fills at most half of the pairs is issued
//     as half tiles;
//   * one persistent CTA pair per two SMs walks the tiles; with `counts` (rows per expert, on the device) the walk goes
//     expert by expert, so the host never waits for the counts;
//   * with both accumulators of a tile in use (all of TMEM) the next tile's MMAs wait for the epilogue, so it gives an accumulator
//     back as soon as its values are in registers, activated and packed to bf16, and stores them under the next main loop: an SM
//     stores about 32 bytes a cycle, 4096 cycles for its 128 KiB of a tile. The fragment form of the TMEM load and a transposing
//     stmatrix turn rows of W into columns of C (gate and up of one value come to the same thread), from a small shared-memory
//     tile 16-byte row pieces go to C. The exchange with shuffles and the stores before the release took 8000 to 9600 cycles of
//     every tile, and the release then waited about 2000 more for the stores; now 800 (plain) and 2500 (SwiGLU, bound by its
//     exponentials and divisions) per accumulator. The main loop runs at the tensor pipe's rate, 1024 cycles per k-block;
//   * what is left of the epilogue is hidden by moving the accumulators against each other (kLead).
// One B200, us, with the epilogue before this one / with it, and the cut unchanged (all of it under the power cap): 32 experts of 1024 rows, 4096 x 7168 SwiGLU 1623 / 1494,
// 7168 x 2048 944 / 752; 8190 x 7168 x 2048 212 / 172,
// 1000 x 14336 x 8192 SwiGLU 209 / 203 (168 with the cuts of gemm_route.hpp).
#pragma once
#include "gemm_skinny.cuh"

namespace purlin {
namespace ragged {

constexpr int kAccStride = 256, kTmemCols = 512;
// Two epilogue warps per quarter of the TMEM lanes (a quarter is all that a warp may read): the drain is exposed, and with one
// each it took twice as long.
constexpr int kEpiWarps = 8, kThreads = 32 * (2 + kEpiWarps);
constexpr int kStagingBytes = kEpiWarps * 2048;       // a 32 x 32 bf16 tile per epilogue warp
constexpr int kBarrierBytes = 256;
constexpr int kMaxExperts = 512;
constexpr int kTableBytes = 2 * (kMaxExperts + 1) * 4;
// k-blocks at either end of a tile that the first accumulator gets before the second one: it is finished, and drained, while the
// second one's last k-blocks run, and the next tile starts with it while the second one is drained. The MMAs of a k-block go into
// one accumulator then, and each waits for the one before (174 cycles instead of 128, measured): longer leads cost more than they
// hide (0 / 1 / 2 / 3 k-blocks, us, 32 experts of 1024 rows: 4096 x 7168 SwiGLU 1541 / 1513 / 1494 / 1507, 7168 x 2048 800 / 771 /
// 752 / 758). A lead holds that many stages.
constexpr int kLead = 2;
constexpr int kBand = 8;                        // column tiles that are in flight together (their X rows stay in L2)

struct alignas(64) Maps { CUtensorMap w, x; };

struct Params {
  int N, K, tokens;        // N: rows of W per expert; tokens: rows of X (with counts: an upper bound of their sum)
  int tileAccs;            // accumulators of a tile: 2 (512 rows of W) or 1 (256)
  int colTiles, maxCols;   // column tiles, and columns of the widest one; with counts an expert has a tile per maxCols rows
  int parts;               // SPLIT: pairs of a cluster
  int stages, narrowStages;            // of so many bytes each, in kRingBytes; narrow: with counts, tiles of kNarrowCols columns
  uint32_t stageBytes, narrowStageBytes;
  int experts;
  const int32_t* counts;   // rows per expert, or null: one group of `tokens` rows
  __nv_bfloat16* C;
  int ldc;
  uint32_t* status;
  uint64_t timeoutNs;
};

PURLIN_D void stCluster16(uint32_t clusterAddress, uint32_t a, uint32_t b, uint32_t c, uint32_t d) {
  asm volatile("st.shared::cluster.v4.u32 [%0], {%1,%2,%3,%4};" ::"r"(clusterAddress), "r"(a), "r"(b), "r"(c), "r"(d) : "memory");
}

// SPLIT: a cluster holds several pairs, which share one tile: each takes a part of its k range, and the partial tiles meet in
// distributed shared memory, in the place of the stages, where each pair finishes every so-many-th chunk of 32 columns, added in the
// order of k. (Through global memory, the last pair to arrive adding them up, the same took 19000 to 45000 cycles instead of about
// 5000.) One tile per cluster, nobody waits for another cluster.
template <bool SWIGLU, bool SPLIT>
__global__ void __launch_bounds__(kThreads, 1) raggedGemmKernel(const __grid_constant__ Maps maps, const __grid_constant__ Params p) {
  extern __shared__ unsigned char smemRaw[];
  const uint32_t rawAddr = tc::smemAddr(smemRaw);
  const uint32_t base = (rawAddr + 1023u) & ~1023u;
  unsigned char* smem = smemRaw + (base - rawAddr);
  const uint32_t xAt = uint32_t(p.tileAccs * kABytes);         // a stage: [W block 0][W block 1, with two accumulators][X: this CTA's half of the columns]
  const uint32_t stagingAll = base + kRingBytes;
  const uint32_t barBase = stagingAll + kStagingBytes;
  auto fullBar = [&](uint32_t s) { return barBase + 8u * s; };
  auto emptyBar = [&](uint32_t s) { return barBase + 8u * (uint32_t(kMaxStages) + s); };
  auto tmemFullBar = [&](int a) { return barBase + 8u * (2u * uint32_t(kMaxStages) + uint32_t(a)); };
  auto tmemEmptyBar = [&](int a) { return barBase + 8u * (2u * uint32_t(kMaxStages) + 2u + uint32_t(a)); };
  unsigned char* tail = smem + kRingBytes + kStagingBytes;
  uint32_t* words = reinterpret_cast<uint32_t*>(tail + 8 * (2 * kMaxStages + 4));
  volatile uint32_t* tmemBaseWord = words;
  volatile int* abortWord = reinterpret_cast<volatile int*>(words + 1);
  volatile uint32_t* narrowWord = words + 2;                          // whether the experts' tiles are narrow
  int* itemStart = reinterpret_cast<int*>(tail + kBarrierBytes);      // [experts + 1] first tile of an expert
  int* rowStart = itemStart + (kMaxExperts + 1);                      // [experts + 1] first row of X of an expert

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t clusterRank = tc::clusterCtaRank(), ctaRank = clusterRank & 1u;
  const int parts = SPLIT ? p.parts : 1, part = SPLIT ? int(clusterRank / 2) : 0;     // pairs that share a tile
  const int pairIdx = int(blockIdx.x) / (2 * parts), numPairs = int(gridDim.x) / (2 * parts);
  const int tileRows = kAccRows * p.tileAccs, wTiles = (p.N + tileRows - 1) / tileRows;
  auto tilesOf = [&](int rows, bool narrow) {
    const int cols = narrow ? kNarrowCols : p.maxCols;
    return p.counts ? (rows + cols - 1) / cols : p.colTiles;
  };

  if (threadIdx.x == 0) {
    for (int s = 0; s < kMaxStages; ++s) { tc::mbarInit(fullBar(s), 1); tc::mbarInit(emptyBar(s), 1); }
    for (int a = 0; a < 2; ++a) { tc::mbarInit(tmemFullBar(a), 1); tc::mbarInit(tmemEmptyBar(a), 2 * kEpiWarps); }   // the warps of both CTAs
    *abortWord = 0;
    tc::mbarFenceInit();
    tc::tmaPrefetchDescriptor(&maps.w);
    tc::tmaPrefetchDescriptor(&maps.x);
  }
  const int kBlocks = (p.K + kBK - 1) / kBK;
  const int kbBegin = int(int64_t(kBlocks) * part / parts), kbEnd = int(int64_t(kBlocks) * (part + 1) / parts);   // this pair's k-blocks
  if (warp == 1) { tc::tmemAllocPair(tc::smemAddr(words), kTmemCols); tc::tmemRelinquishPair(); }
  tc::gridDependencyWait();                                    // from here on memory that earlier kernels write may be read
  if (warp == 2) {
    // rows and tiles of every expert, as running sums: 32 experts per step
    const uint32_t limit = uint32_t(p.tokens);
    uint32_t rows0 = 0;
    int items0 = 0;
    // Narrow tiles have room for a fifth stage, but an expert of many rows then reads its weights once for every 64 of them: they are taken
    // where they are at most an eighth more tiles (MoE block 7168 / 2048 of 32 experts, one of which gets the most rows, us, wide / narrow:
    // average 32, most 128 497 / 489; 19, 300 493 / 484; 40, 640 498 / 548; 40, 654 501 / 556).
    bool narrow = false;
    if (p.counts) {
      uint32_t few = 0, many = 0;
      for (int e = lane; e < p.experts; e += 32) {
        const int r = int(skinny::groupRowsOf(p.counts[e], limit));
        few += uint32_t(tilesOf(r, false));
        many += uint32_t(tilesOf(r, true));
      }
      few = __reduce_add_sync(0xffffffffu, few);
      many = __reduce_add_sync(0xffffffffu, many);
      narrow = uint64_t(many) * 8 <= uint64_t(few) * 9;
    }
    if (lane == 0) *narrowWord = narrow ? 1u : 0u;
    for (int e0 = 0; e0 < p.experts; e0 += 32) {
      const int e = e0 + lane;
      uint32_t sum = e < p.experts ? (p.counts ? skinny::groupRowsOf(p.counts[e], limit) : limit) : 0u;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) { const uint32_t v = __shfl_up_sync(0xffffffffu, sum, o); if (lane >= o) sum = skinny::addRows(sum, v, limit); }
      const uint32_t before = __shfl_up_sync(0xffffffffu, sum, 1);
      const int first = int(lane ? skinny::addRows(rows0, before, limit) : rows0), end = int(skinny::addRows(rows0, sum, limit));
      const int r = end - first;
      const int n = r > 0 ? tilesOf(r, narrow) * wTiles : 0;
      int items = n;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) { const int v = __shfl_up_sync(0xffffffffu, items, o); if (lane >= o) items += v; }
      if (e < p.experts) { rowStart[e] = first; itemStart[e] = items0 + items - n; rowStart[e + 1] = end; itemStart[e + 1] = items0 + items; }
      rows0 = skinny::addRows(rows0, __shfl_sync(0xffffffffu, sum, 31), limit);
      items0 += __shfl_sync(0xffffffffu, items, 31);
      __syncwarp();
    }
  }
  tc::fenceBeforeThreadSync();
  __syncthreads();
  tc::clusterSync();                                           // the pair's barriers exist before any remote arrival
  tc::fenceAfterThreadSync();
  tc::gridLaunchDependents();
  const uint32_t tmemBase = *tmemBaseWord;
  const bool narrow = *narrowWord != 0;
  const uint32_t stages = uint32_t(narrow ? p.narrowStages : p.stages), stageBytes = narrow ? p.narrowStageBytes : p.stageBytes;
  const uint32_t leaderBars = tc::mapToCta(barBase, clusterRank & ~1u), pairMask = 3u << (clusterRank & ~1u);
  const int numTiles = itemStart[p.experts], rest = numTiles % numPairs;
  // whole tiles; the others count as two items each
  const int fullItems = !SPLIT && p.tileAccs == 2 && 2 * rest <= numPairs ? numTiles - rest : numTiles;
  const int numItems = fullItems + 2 * (numTiles - fullItems);

  // work item -> expert, first row of X, valid columns, columns of the MMA, first row of W inside the expert, accumulators
  struct Item { int expert, row0, cols, count, w0, accs; };
  int expert = 0;                                              // items are visited in ascending order
  auto itemOf = [&](int it) {
    const int tile = it < fullItems ? it : fullItems + ((it - fullItems) >> 1);
    while (tile >= itemStart[expert + 1]) ++expert;
    Item m;
    m.expert = expert;
    const int rows = rowStart[expert + 1] - rowStart[expert], tiles = tilesOf(rows, narrow);
    const int i = tile - itemStart[expert], units = (rows + 31) / 32;
    int first = 0, width = units;                              // of the column tile, in units of 32 (steps of an MMA of a pair)
    m.w0 = i * tileRows;
    if (tiles > 1) {                                           // (a few divisions that a stream of small tiles would notice: decode 6 %)
      const int perBand = kBand * wTiles, band = i / perBand, within = i - band * perBand;
      const int inBand = min(tiles - band * kBand, kBand), wTile = within / inBand;
      const int col = band * kBand + within - wTile * inBand;
      m.w0 = wTile * tileRows;
      // the rows of X are shared out evenly over the column tiles
      const int each = units / tiles, more = units - each * tiles;
      first = col * each + min(col, more);
      width = each + (col < more ? 1 : 0);
    }
    m.cols = 32 * width;
    m.row0 = rowStart[expert] + 32 * first;
    m.count = min(m.cols, rows - 32 * first);
    m.accs = p.tileAccs == 2 && m.w0 + kAccRows < p.N ? 2 : 1;
    if (it >= fullItems) {                    // half a tile: 256 rows of W (none, when the tile has no second half)
      const int half = (it - fullItems) & 1;
      m.accs = half < m.accs ? 1 : 0;
      m.w0 += half * kAccRows;
    }
    return m;
  };
  auto forItems = [&](auto&& body) {
    for (int it = pairIdx; it < numItems; it += numPairs) {
      const Item m = itemOf(it);
      if (m.accs && !body(m)) return;
    }
  };
  // One accumulator alone (a tile of 256 rows of W, half a tile): its columns are two chains of MMAs, the two halves in turn, because
  // MMAs into the same columns wait for one another. The pair supplies the columns of each MMA in equal shares, so the rows of X are
  // loaded in quarters then: CTA 0 the first and the third, CTA 1 the others.
  auto inHalves = [&](const Item& m) { return m.accs == 1 && m.cols % 128 == 0; };

  // The pairs' main loops are over, and a wait that gave up in one of them is known to all: they learn of it through their abort words.
  auto agree = [&](bool ok) {
    if (!ok) {
      const uint32_t word = tc::smemAddr(words + 1);
      for (int q = 0; q < 2 * parts; ++q) asm volatile("st.shared::cluster.u32 [%0], %1;" ::"r"(tc::mapToCta(word, uint32_t(q))), "r"(1) : "memory");
    }
    __syncwarp();
    tc::clusterSync();
  };

  if (warp == 0) {
    if (lane == 0) {
      uint32_t st = 0, ph = 0;
      bool ok = true;
      forItems([&](const Item& m) {
        const int half = m.cols / 2, loads = (half + kXBox - 1) / kXBox;
        const bool quarters = inHalves(m);
        const int wRow = m.expert * p.N + m.w0 + int(ctaRank) * kBM;
        const int xRow = m.row0 + int(ctaRank) * (quarters ? half / 2 : half), jump = quarters ? half / 2 : 0;
        const uint32_t bytes = uint32_t(2 * (m.accs * kABytes + loads * kXBox * kBK * 2));
        for (int kb = kbBegin; kb < kbEnd; ++kb) {
          ok = tc::mbarWait(emptyBar(st), ph ^ 1, abortWord, p.timeoutNs);
          if (!ok) { skinny::recordTimeout(p.status, 1, m.w0, kb); break; }
          const uint32_t sW = base + st * stageBytes, sX = sW + xAt;
          const uint32_t leaderFull = leaderBars + 8u * st;
          if (ctaRank == 0) tc::mbarExpectTx(fullBar(st), bytes);        // both CTAs' bytes are credited to CTA 0's barrier
          tc::tmaLoad2dPair(sW, &maps.w, kb * kBK, wRow, leaderFull);
          if (m.accs == 2) tc::tmaLoad2dPair(sW + kABytes, &maps.w, kb * kBK, wRow + 2 * kBM, leaderFull);
          for (int i = 0; i < loads; ++i)
            tc::tmaLoad2dPair(sX + uint32_t(i * kXBox * kBK * 2), &maps.x, kb * kBK, xRow + i * kXBox + (2 * i >= loads ? jump : 0), leaderFull);
          if (++st == stages) { st = 0; ph ^= 1; }
        }
        return ok;
      });
    }
  } else if (warp == 1) {
    if (lane == 0 && ctaRank == 0) {
      // descriptors differ only in their 14-bit start address: one constant upper half, the lower halves of the current stage
      const uint64_t descW0 = tc::smemDescSw128(base), descX0 = tc::smemDescSw128(base + xAt);
      const uint32_t high = uint32_t(descW0 >> 32), stageStep = stageBytes >> 4;
      auto desc = [&](uint32_t low) { return uint64_t(high) << 32 | low; };
      uint32_t st = 0, ph = 0, at = 0, use = 0, single = 0;    // at: offset of stage st; bit a of `use`: parity of the uses of accumulator a so far
      bool ok = true;
      const int n = kbEnd - kbBegin;
      forItems([&](const Item& m) {
        const bool two = m.accs == 2, halves = inHalves(m);
        const uint32_t idesc = tc::instrDescBf16(uint32_t(halves ? m.cols / 2 : m.cols), uint32_t(2 * kBM));
        const int a0 = two ? 0 : int(single++ & 1);            // tiles of one accumulator alternate between the two
        ok = tc::mbarWait(tmemEmptyBar(a0), ((use >> a0) & 1) ^ 1, abortWord, p.timeoutNs);
        if (!ok) { skinny::recordTimeout(p.status, 2, m.w0, a0); return false; }
        uint32_t accumulate = 0;
        // One thread feeds the tensor cores of two SMs (an MMA takes about 128 cycles), so the loops over the stages hold
        // nothing but waits, MMAs and commits: which accumulators there are is decided outside of them.
        auto landed = [&](int kb) {                            // the k-block in the current stage
          ok = tc::mbarWait(fullBar(st), ph, abortWord, p.timeoutNs);
          if (!ok) { skinny::recordTimeout(p.status, 3, m.w0, kb); return false; }
          tc::fenceAfterThreadSync();
          return true;
        };
        auto release = [&]() {                                 // of the current stage, once the MMAs issued so far have read it
          tc::mmaCommitPairs(emptyBar(st), pairMask);
        };
        auto advance = [&]() {
          at += stageStep;
          if (++st == stages) { st = 0; at = 0; ph ^= 1; }
        };
        auto complete = [&](int a) {                           // the epilogue may read accumulator a
          tc::mmaCommitPairs(tmemFullBar(a), pairMask);
        };
        const uint32_t w0 = uint32_t(descW0), w1 = w0 + (kABytes >> 4), x0 = uint32_t(descX0);
        const uint32_t d0 = tmemBase + uint32_t(a0) * kAccStride, d1 = tmemBase + kAccStride;
        if (two) {
          const int ends = min(kLead, n / 2);
          auto oneThenOther = [&](int kb0, bool last) {
            const uint32_t st0 = st, ph0 = ph, at0 = at;
            for (int i = 0; i < ends && ok; ++i) {
              if (!landed(kb0 + i)) return;
#pragma unroll
              for (int k = 0; k < kBK / 16; ++k) { tc::mmaPair(d0, desc(w0 + at + 2 * k), desc(x0 + at + 2 * k), idesc, accumulate); accumulate = 1; }
              advance();
            }
            if (last) complete(0);
            else ok = tc::mbarWait(tmemEmptyBar(1), ((use >> 1) & 1) ^ 1, abortWord, p.timeoutNs);
            if (!ok) { skinny::recordTimeout(p.status, 2, m.w0, 1); return; }
            st = st0; ph = ph0; at = at0;
            for (int i = 0; i < ends; ++i) {
#pragma unroll
              for (int k = 0; k < kBK / 16; ++k) tc::mmaPair(d1, desc(w1 + at + 2 * k), desc(x0 + at + 2 * k), idesc, uint32_t(last || i || k));
              release();
              advance();
            }
          };
          oneThenOther(0, false);
          for (int kb = ends; kb < n - ends && ok; ++kb) {
            if (!landed(kb)) break;
#pragma unroll
            for (int k = 0; k < kBK / 16; ++k) {
              tc::mmaPair(d0, desc(w0 + at + 2 * k), desc(x0 + at + 2 * k), idesc, accumulate);
              tc::mmaPair(d1, desc(w1 + at + 2 * k), desc(x0 + at + 2 * k), idesc, accumulate);
              accumulate = 1;
            }
            release();
            advance();
          }
          if (ok) oneThenOther(n - ends, true);
          if (ok) { complete(1); use ^= 3u; }
        } else if (halves) {
          const uint32_t dh = d0 + uint32_t(m.cols / 2), xh = x0 + uint32_t(m.cols / 4 * kBK * 2 >> 4);
          for (int kb = 0; kb < n; ++kb) {
            if (!landed(kb)) break;
#pragma unroll
            for (int k = 0; k < kBK / 16; ++k) {
              tc::mmaPair(d0, desc(w0 + at + 2 * k), desc(x0 + at + 2 * k), idesc, accumulate);
              tc::mmaPair(dh, desc(w0 + at + 2 * k), desc(xh + at + 2 * k), idesc, accumulate);
              accumulate = 1;
            }
            release();
            advance();
          }
        } else {
          for (int kb = 0; kb < n; ++kb) {
            if (!landed(kb)) break;
#pragma unroll
            for (int k = 0; k < kBK / 16; ++k) { tc::mmaPair(d0, desc(w0 + at + 2 * k), desc(x0 + at + 2 * k), idesc, accumulate); accumulate = 1; }
            release();
            advance();
          }
        }
        if (ok && !two) { complete(a0); use ^= 1u << a0; }
        return ok;
      });
    }
  } else {
    // ------------------------------- epilogue -------------------------------
    constexpr int kOut = SWIGLU ? 16 : 32;                     // output columns of this warp's 32 rows of W
    constexpr int kPitch = kOut * 2;                           // bytes of a token's row in the staging tile
    constexpr int kChunks = kMaxCols / 64, kHeld = kOut / 2;   // per accumulator of a warp: 32-column chunks, packed registers of each
    constexpr int kPieces = kOut / 8, kRowsPer = 32 / kPieces; // 16-byte pieces of such a row; rows per access of the warp
    const int quarter = warp & 3;                              // a warp may only touch TMEM lanes [32 * (warp % 4), +32)
    const int outCols = SWIGLU ? p.N / 2 : p.N;
    const int group = (warp - 2) / 4;                          // two warps per quarter share the columns, 32 by 32
    const uint32_t buf = stagingAll + uint32_t(warp - 2) * 2048u;
    // where 16-byte piece `piece` of token row `row` lies in the staging tile: rotated so that neither the eight rows of a
    // transposed store nor the reads meet in a bank
    auto stagedAt = [&](int row, int piece) { return buf + uint32_t(row * kPitch + ((piece ^ ((row * kPitch >> 7) & (kPieces - 1))) << 4)); };
    const int piece = lane % kPieces, rr = lane / kPieces;
    auto f = [](uint32_t v) { return __uint_as_float(v); };
    // 32 columns (tokens) of this warp's 32 rows of W, fragments of rows 0-15 and of rows 16-31 -> activated and packed
    auto activate = [&](const uint32_t (&lo)[16], const uint32_t (&hi)[16], uint32_t (&h)[kHeld]) {
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        if constexpr (SWIGLU)                                  // rows 0-15 are gate, 16-31 up, of the same 16 output columns
          h[i] = skinny::pack2(skinny::siluOf(f(lo[2 * i])) * f(hi[2 * i]), skinny::siluOf(f(lo[2 * i + 1])) * f(hi[2 * i + 1]));
        else {
          h[i] = skinny::pack2(f(lo[2 * i]), f(lo[2 * i + 1]));
          h[8 + i] = skinny::pack2(f(hi[2 * i]), f(hi[2 * i + 1]));
        }
      }
    };
    // ... -> C, turned around on the way through the staging tile: rows of W become columns of C. c: first column of the chunk.
    auto store = [&](const Item& m, int block, int c, const uint32_t (&h)[kHeld]) {
      const int wRow = m.w0 + block * kAccRows + int(ctaRank) * kBM + quarter * 32;  // of lane 0
      const int n0 = (SWIGLU ? wRow / 2 : wRow) + piece * 8;
      const bool colOk = n0 + 8 <= outCols;
      __nv_bfloat16* out = p.C + size_t(m.row0) * p.ldc + n0;
      if constexpr (SWIGLU) {
#pragma unroll
        for (int i = 0; i < 4; i += 2)
          tc::stMatrixTransposed4(stagedAt(8 * (i + (lane >> 4)) + (lane & 7), (lane >> 3) & 1), h[2 * i], h[2 * i + 1], h[2 * i + 2], h[2 * i + 3]);
      } else {
#pragma unroll
        for (int i = 0; i < 4; ++i)
          tc::stMatrixTransposed4(stagedAt(8 * i + (lane & 7), lane >> 3), h[2 * i], h[2 * i + 1], h[8 + 2 * i], h[8 + 2 * i + 1]);
      }
      __syncwarp();
#pragma unroll
      for (int i = 0; i < kPieces; ++i) {
        Vec16 v;
        asm volatile("ld.shared.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(v.x[0]), "=r"(v.x[1]), "=r"(v.x[2]), "=r"(v.x[3]) : "r"(stagedAt(i * kRowsPer + rr, piece)) : "memory");
        const int row = c + i * kRowsPer + rr;
        if (colOk && row < m.count) st16(out + size_t(row) * p.ldc, v);
      }
      __syncwarp();                                            // the tile has been read before the next chunk fills it
    };
    auto load = [&](int a, int c, uint32_t (&lo)[16], uint32_t (&hi)[16]) {
      const uint32_t taddr = tmemBase + (uint32_t(quarter * 32) << 16) + uint32_t(a) * kAccStride + uint32_t(c);
      tc::tmemLoadFragments(taddr, lo);
      tc::tmemLoadFragments(taddr + (16u << 16), hi);
      tc::tmemLoadWaitFor(lo);
      tc::tmemLoadWaitFor(hi);
    };
    uint32_t use = 0, single = 0;                              // as in the MMA warp
    bool ok = true;
    auto finished = [&](const Item& m, int a) {
      ok = tc::mbarWait(tmemFullBar(a), (use >> a) & 1, abortWord, p.timeoutNs);
      ok = __all_sync(0xffffffffu, ok);
      if (!ok) { if (lane == 0) skinny::recordTimeout(p.status, 5, m.w0, a); return false; }
      use ^= 1u << a;
      tc::fenceAfterThreadSync();
      return true;
    };
    if constexpr (!SPLIT) {
      forItems([&](const Item& m) {
        const int a0 = m.accs == 2 ? 0 : int(single++ & 1);
        // into registers, activated and packed; the accumulator goes back to the MMA warp
        uint32_t held[2][kChunks][kHeld];
#pragma unroll
        for (int b = 0; b < 2; ++b) {
          if (b >= m.accs || !ok || !finished(m, a0 + b)) continue;
#pragma unroll
          for (int j = 0; j < kChunks; ++j) {
            if (group * 32 + j * 64 >= m.count) continue;
            uint32_t lo[16], hi[16];
            load(a0 + b, group * 32 + j * 64, lo, hi);
            activate(lo, hi, held[b][j]);
          }
          tc::fenceBeforeThreadSync();
          __syncwarp();
          if (lane == 0) tc::mbarArriveClusterTmem(leaderBars + 8u * (2u * uint32_t(kMaxStages) + 2u + uint32_t(a0 + b)));
        }
        if (!ok) return false;
#pragma unroll
        for (int b = 0; b < 2; ++b)
#pragma unroll
          for (int j = 0; j < kChunks; ++j)
            if (b < m.accs && group * 32 + j * 64 < m.count) store(m, b, group * 32 + j * 64, held[b][j]);
        return true;
      });
    } else {
      // (one item, so accumulator b is b) a chunk c of accumulator b is finished by pair c % parts, there it has a slot for every other
      // pair; a warp's 32 x 32 values lie in it as the fragments lie in registers, 512 bytes per access of the warp
      const int slots = (kMaxCols / 32 + parts - 1) / parts;
      auto slotOf = [&](int from, int at, int b, int c) {
        const int q = from < at ? from : from - 1;
        return base + uint32_t((((q * 2 + b) * slots + c / parts) * 4 + quarter) * 4096 + lane * 16);
      };
      forItems([&](const Item& m) { for (int b = 0; b < m.accs && finished(m, b); ++b) {} return ok; });
      agree(ok);
      forItems([&](const Item& m) {
        for (int b = 0; b < m.accs; ++b)
          for (int c = group; c * 32 < m.count; c += 2) {
            if (c % parts == part || *abortWord) continue;
            uint32_t lo[16], hi[16];
            load(b, c * 32, lo, hi);
            const uint32_t to = tc::mapToCta(slotOf(part, c % parts, b, c), uint32_t(c % parts) * 2 + ctaRank);
#pragma unroll
            for (int i = 0; i < 4; ++i) {
              stCluster16(to + i * 512, lo[4 * i], lo[4 * i + 1], lo[4 * i + 2], lo[4 * i + 3]);
              stCluster16(to + (i + 4) * 512, hi[4 * i], hi[4 * i + 1], hi[4 * i + 2], hi[4 * i + 3]);
            }
          }
        return true;
      });
      __syncwarp();
      tc::clusterSync();
      forItems([&](const Item& m) {
        for (int b = 0; b < m.accs; ++b)
          for (int c = group; c * 32 < m.count; c += 2) {
            if (c % parts != part || *abortWord) continue;
            uint32_t lo[16], hi[16], own[2][16], h[kHeld];
            load(b, c * 32, own[0], own[1]);
#pragma unroll
            for (int i = 0; i < 16; ++i) lo[i] = hi[i] = 0u;
            auto add = [&](uint32_t& to, uint32_t x) { to = __float_as_uint(f(to) + f(x)); };
#pragma unroll 1
            for (int q = 0; q < parts; ++q) {
              if (q == part) {
#pragma unroll
                for (int i = 0; i < 16; ++i) { add(lo[i], own[0][i]); add(hi[i], own[1][i]); }
              } else {
                const uint32_t from = slotOf(q, part, b, c);
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                  uint32_t v[4], u[4];
                  asm volatile("ld.shared.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]) : "r"(from + i * 512) : "memory");
                  asm volatile("ld.shared.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(u[0]), "=r"(u[1]), "=r"(u[2]), "=r"(u[3]) : "r"(from + (i + 4) * 512) : "memory");
#pragma unroll
                  for (int e = 0; e < 4; ++e) { add(lo[4 * i + e], v[e]); add(hi[4 * i + e], u[e]); }
                }
              }
            }
            activate(lo, hi, h);
            store(m, b, c * 32, h);
          }
        return true;
      });
    }
  }
  if (SPLIT && warp < 2) { agree(*abortWord == 0); __syncwarp(); tc::clusterSync(); }      // the two barriers of the exchange

  if (*abortWord) tc::landingPause();   // copies already in flight land before shared memory and TMEM go away
  __syncwarp();
  tc::fenceBeforeThreadSync();
  tc::clusterSync();                    // neither CTA frees TMEM the pair's MMA still writes
  if (warp == 1) tc::tmemDeallocPair(tmemBase, kTmemCols);
}

}  // namespace ragged
}  // namespace purlin
