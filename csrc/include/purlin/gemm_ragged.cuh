// GEMM for any number of activation rows, plain or per expert: C[T, N] = X[T, K] * W[N, K]^T on CTA pairs.
//
// What bounds it is the tensor pipe, and the loss it removes is padding: the rows of X (a prompt chunk, the rows of an
// expert) are no multiple of a 256- or 512-row tile. So W fills the rows of the MMA (its row count is a multiple of the
// tile in practice) and the rows of X are the columns, whose number may be any multiple of 32: T rows are cut into
// column tiles of `tileCols` and one narrower tile for the remainder.
//   * a tile is 512 rows of W (two accumulators of a CTA pair, 256 rows each) x up to 256 rows of X; the two accumulators
//     share the X operand, which the tensor pipe rewards (see gemm_sm100.cu). A last wave that fills at most half of the
//     pairs is issued as half tiles (256 rows of W);
//   * one persistent CTA pair per two SMs walks the tiles; with `counts` (rows per expert, on the device) the walk goes
//     expert by expert, so the host never waits for the counts;
//   * the epilogue turns the accumulator around: TMEM lanes are rows of W, so neighbouring lanes pair up (one shuffle per
//     two values) and write rows of X into a small shared-memory tile, from which 16-byte row pieces go to C.
#pragma once
#include <type_traits>

#include "gemm_skinny.cuh"

namespace purlin {
namespace ragged {

constexpr int kBM = 128, kBK = 64, kMaxCols = 256;
constexpr int kABytes = kBM * kBK * 2;
constexpr int kTileRows = 512;                  // rows of W per tile: 2 accumulators x 2 CTAs x 128
constexpr int kAccStride = 256, kTmemCols = 512;
// Four epilogue warps per accumulator: with both accumulators of a tile in use the epilogue is exposed, and eight warps halve it
// (four / eight warps, one B200: 3000 x 7168 x 2048 77.5 / 73.3 us, 1500 x 4096 x 4096 SwiGLU 51.1 / 46.9, 32 experts of 1024
// rows 1748 + 1151 / 1631 + 1130).
constexpr int kEpiWarps = 8, kThreads = 32 * (2 + kEpiWarps);
constexpr int kStagingBytes = kEpiWarps * 2048;       // a 32 x 32 bf16 tile per epilogue warp
constexpr int kBarrierBytes = 256;
constexpr int kMaxExperts = 512;
constexpr int kTableBytes = 2 * (kMaxExperts + 1) * 4;
constexpr int kMaxStages = 6;
constexpr int kBand = 8;                        // column tiles that are in flight together (their X rows stay in L2)

struct alignas(64) Maps { CUtensorMap w, x; };

struct Params {
  int N, K, tokens;        // N: rows of W per expert; tokens: rows of X (with counts: an upper bound of their sum)
  int tileCols;            // columns of a tile: a multiple of 64, at most 256
  int xBox;                // rows of one X load
  int stages;
  int experts;
  const int32_t* counts;   // rows per expert, or null: one group of `tokens` rows
  __nv_bfloat16* C;
  int ldc;
  uint32_t* status;
  uint64_t timeoutNs;
};

template <bool SWIGLU>
__global__ void __launch_bounds__(kThreads, 1) raggedGemmKernel(const __grid_constant__ Maps maps, const __grid_constant__ Params p) {
  extern __shared__ unsigned char smemRaw[];
  const uint32_t rawAddr = tc::smemAddr(smemRaw);
  const uint32_t base = (rawAddr + 1023u) & ~1023u;
  unsigned char* smem = smemRaw + (base - rawAddr);
  constexpr int kXBytes = kMaxCols / 2 * kBK * 2;              // this CTA's half of the columns
  constexpr uint32_t kStageBytes = 2 * kABytes + kXBytes;      // [W block 0][W block 1][X]
  const uint32_t stagingAll = base + uint32_t(p.stages) * kStageBytes;
  const uint32_t barBase = stagingAll + kStagingBytes;
  auto fullBar = [&](uint32_t s) { return barBase + 8u * s; };
  auto emptyBar = [&](uint32_t s) { return barBase + 8u * (uint32_t(p.stages) + s); };
  auto tmemFullBar = [&](int a) { return barBase + 8u * (2u * uint32_t(p.stages) + uint32_t(a)); };
  auto tmemEmptyBar = [&](int a) { return barBase + 8u * (2u * uint32_t(p.stages) + 2u + uint32_t(a)); };
  unsigned char* tail = smem + size_t(p.stages) * kStageBytes + kStagingBytes;
  uint32_t* words = reinterpret_cast<uint32_t*>(tail + 8 * (2 * p.stages + 4));
  volatile uint32_t* tmemBaseWord = words;
  volatile int* abortWord = reinterpret_cast<volatile int*>(words + 1);
  int* itemStart = reinterpret_cast<int*>(tail + kBarrierBytes);      // [experts + 1] first tile of an expert
  int* rowStart = itemStart + (kMaxExperts + 1);                      // [experts + 1] first row of X of an expert

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t ctaRank = tc::clusterCtaRank();
  const int pairIdx = int(blockIdx.x) / 2, numPairs = int(gridDim.x) / 2;
  const int wTiles = (p.N + kTileRows - 1) / kTileRows;
  auto tilesOf = [&](int rows) { return (rows + p.tileCols - 1) / p.tileCols; };

  if (threadIdx.x == 0) {
    for (int s = 0; s < p.stages; ++s) { tc::mbarInit(fullBar(s), 1); tc::mbarInit(emptyBar(s), 1); }
    for (int a = 0; a < 2; ++a) { tc::mbarInit(tmemFullBar(a), 1); tc::mbarInit(tmemEmptyBar(a), kEpiWarps); }   // 4 warps in each CTA
    *abortWord = 0;
    tc::mbarFenceInit();
    tc::tmaPrefetchDescriptor(&maps.w);
    tc::tmaPrefetchDescriptor(&maps.x);
  }
  if (warp == 1) { tc::tmemAllocPair(tc::smemAddr(words), kTmemCols); tc::tmemRelinquishPair(); }
  tc::gridDependencyWait();                                    // from here on memory that earlier kernels write may be read
  if (warp == 2) {
    // rows and tiles of every expert, as running sums: 32 experts per step
    const uint32_t limit = uint32_t(p.tokens);
    uint32_t rows0 = 0;
    int items0 = 0;
    for (int e0 = 0; e0 < p.experts; e0 += 32) {
      const int e = e0 + lane;
      uint32_t sum = e < p.experts ? (p.counts ? skinny::groupRowsOf(p.counts[e], limit) : limit) : 0u;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) { const uint32_t v = __shfl_up_sync(0xffffffffu, sum, o); if (lane >= o) sum = skinny::addRows(sum, v, limit); }
      const uint32_t before = __shfl_up_sync(0xffffffffu, sum, 1);
      const int first = int(lane ? skinny::addRows(rows0, before, limit) : rows0), end = int(skinny::addRows(rows0, sum, limit));
      const int r = end - first;
      const int n = r > 0 ? tilesOf(r) * wTiles : 0;
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
  const uint32_t leaderBars = tc::mapToCta(barBase, 0), peerBars = tc::mapToCta(barBase, 1);
  const int numTiles = itemStart[p.experts], rest = numTiles % numPairs;
  const int fullItems = 2 * rest <= numPairs ? numTiles - rest : numTiles;        // whole tiles; the others count as two items each
  const int numItems = fullItems + 2 * (numTiles - fullItems);
  const int kBlocks = (p.K + kBK - 1) / kBK;

  // work item -> expert, first row of X, valid columns, columns of the MMA, first row of W inside the expert, accumulators
  struct Item { int expert, row0, cols, count, w0, accs; };
  int expert = 0;                                              // items are visited in ascending order
  auto itemOf = [&](int it) {
    const int tile = it < fullItems ? it : fullItems + ((it - fullItems) >> 1);
    while (tile >= itemStart[expert + 1]) ++expert;
    Item m;
    m.expert = expert;
    const int rows = rowStart[expert + 1] - rowStart[expert], tiles = tilesOf(rows);
    const int i = tile - itemStart[expert], perBand = kBand * wTiles, band = i / perBand, within = i - band * perBand;
    const int inBand = min(tiles - band * kBand, kBand);
    const int col = band * kBand + within % inBand;
    m.w0 = within / inBand * kTileRows;
    m.row0 = rowStart[expert] + col * p.tileCols;
    m.count = min(p.tileCols, rows - col * p.tileCols);
    m.cols = (m.count + 31) / 32 * 32;                         // steps of 32, as the MMA of a pair wants them
    m.accs = m.w0 + kTileRows / 2 < p.N ? 2 : 1;
    if (it >= fullItems) {                                     // half a tile: 256 rows of W (none, when the tile has no second half)
      const int half = (it - fullItems) & 1;
      m.accs = half < m.accs ? 1 : 0;
      m.w0 += half * (kTileRows / 2);
    }
    return m;
  };

  if (warp == 0) {
    if (lane == 0) {
      uint32_t st = 0, ph = 0;
      bool ok = true;
      for (int it = pairIdx; it < numItems && ok; it += numPairs) {
        const Item m = itemOf(it);
        if (m.accs == 0) continue;
        const int half = m.cols / 2, loads = (half + p.xBox - 1) / p.xBox;
        const int wRow = m.expert * p.N + m.w0 + int(ctaRank) * kBM, xRow = m.row0 + int(ctaRank) * half;
        const uint32_t bytes = uint32_t(2 * (m.accs * kABytes + loads * p.xBox * kBK * 2));
        for (int kb = 0; kb < kBlocks; ++kb) {
          ok = tc::mbarWait(emptyBar(st), ph ^ 1, abortWord, p.timeoutNs);
          if (!ok) { skinny::recordTimeout(p.status, 1, it, kb); break; }
          const uint32_t sW = base + st * kStageBytes, sX = sW + 2 * kABytes;
          const uint32_t leaderFull = leaderBars + 8u * st;
          if (ctaRank == 0) tc::mbarExpectTx(fullBar(st), bytes);        // both CTAs' bytes are credited to CTA 0's barrier
          tc::tmaLoad2dPair(sW, &maps.w, kb * kBK, wRow, leaderFull);
          if (m.accs == 2) tc::tmaLoad2dPair(sW + kABytes, &maps.w, kb * kBK, wRow + 2 * kBM, leaderFull);
          for (int i = 0; i < loads; ++i)
            tc::tmaLoad2dPair(sX + uint32_t(i * p.xBox * kBK * 2), &maps.x, kb * kBK, xRow + i * p.xBox, leaderFull);
          if (++st == uint32_t(p.stages)) { st = 0; ph ^= 1; }
        }
      }
    }
  } else if (warp == 1) {
    if (lane == 0 && ctaRank == 0) {
      const uint64_t descW0 = tc::smemDescSw128(base), descX0 = tc::smemDescSw128(base + 2 * kABytes);
      uint32_t st = 0, ph = 0, use0 = 0, use1 = 0;
      bool ok = true;
      for (int it = pairIdx; it < numItems && ok; it += numPairs) {
        const Item m = itemOf(it);
        if (m.accs == 0) continue;
        const uint32_t idesc = tc::instrDescBf16(uint32_t(m.cols), uint32_t(2 * kBM));
        const bool two = m.accs == 2;
        ok = tc::mbarWait(tmemEmptyBar(0), (use0 & 1) ^ 1, abortWord, p.timeoutNs);
        if (ok && two) ok = tc::mbarWait(tmemEmptyBar(1), (use1 & 1) ^ 1, abortWord, p.timeoutNs);
        if (!ok) { skinny::recordTimeout(p.status, 2, it, 0); break; }
        // One thread feeds the tensor cores of two SMs (an MMA takes about 128 cycles), so the loop over the stages holds
        // nothing but waits, MMAs and commits: which accumulators there are is decided outside of it.
        auto issue = [&](auto both) {
          uint32_t accumulate = 0;
          for (int kb = 0; kb < kBlocks; ++kb) {
            ok = tc::mbarWait(fullBar(st), ph, abortWord, p.timeoutNs);
            if (!ok) { skinny::recordTimeout(p.status, 3, it, kb); break; }
            tc::fenceAfterThreadSync();
            const uint64_t step = uint64_t(st * (kStageBytes >> 4));
#pragma unroll
            for (int k = 0; k < kBK / 16; ++k) {
              tc::mmaPair(tmemBase, descW0 + step + 2 * k, descX0 + step + 2 * k, idesc, accumulate);
              if constexpr (decltype(both)::value) tc::mmaPair(tmemBase + kAccStride, descW0 + step + (kABytes >> 4) + 2 * k, descX0 + step + 2 * k, idesc, accumulate);
              accumulate = 1;
            }
            tc::mmaCommitPair(leaderBars + 8u * (uint32_t(p.stages) + st));
            tc::mmaCommitPair(peerBars + 8u * (uint32_t(p.stages) + st));
            if (++st == uint32_t(p.stages)) { st = 0; ph ^= 1; }
          }
        };
        if (two) issue(std::true_type{}); else issue(std::false_type{});
        if (ok) {
          for (int a = 0; a < m.accs; ++a) {
            tc::mmaCommitPair(leaderBars + 8u * (2u * uint32_t(p.stages) + uint32_t(a)));
            tc::mmaCommitPair(peerBars + 8u * (2u * uint32_t(p.stages) + uint32_t(a)));
          }
          ++use0;
          if (two) ++use1;
        }
      }
    }
  } else {
    // ------------------------------- epilogue -------------------------------
    constexpr int kOut = SWIGLU ? 16 : 32;                     // output columns of this warp's 32 rows of W
    constexpr int kPitch = kOut * 2;                           // bytes of a token's row in the staging tile
    const int quarter = warp & 3;                              // a warp may only touch TMEM lanes [32 * (warp % 4), +32)
    const int outCols = SWIGLU ? p.N / 2 : p.N;
    const int a = (warp - 2) / 4;                              // this warp's accumulator
    const uint32_t buf = stagingAll + uint32_t(warp - 2) * 2048u;
    uint32_t use = 0;
    bool ok = true;
    for (int it = pairIdx; it < numItems && ok; it += numPairs) {
      const Item m = itemOf(it);
      if (a < m.accs) {
        ok = tc::mbarWait(tmemFullBar(a), use & 1, abortWord, p.timeoutNs);
        ok = __all_sync(0xffffffffu, ok);
        if (!ok) { if (lane == 0) skinny::recordTimeout(p.status, 5, it, a); break; }
        ++use;
        tc::fenceAfterThreadSync();
        const uint32_t taddr = tmemBase + (uint32_t(quarter * 32) << 16) + uint32_t(a) * kAccStride;
        const int wRow = m.w0 + a * 2 * kBM + int(ctaRank) * kBM + quarter * 32;     // of lane 0
        const int n0 = SWIGLU ? wRow / 2 : wRow;
        __nv_bfloat16* out = p.C + size_t(m.row0) * p.ldc + n0;

        // 32 columns (tokens) of this warp's 32 rows of W -> rows of C
        auto drain = [&](const uint32_t (&r)[32], int c) {
          if constexpr (SWIGLU) {
            // lanes 0-15 hold gate, 16-31 up, of the same 16 output columns: the lower half finishes tokens t and t + 1, the
            // upper half t + 2 and t + 3; then neighbouring lanes pair up so that each writes two columns of one token
            const bool low = lane < 16, even = (lane & 1) == 0;
#pragma unroll
            for (int t = 0; t < 32; t += 4) {
              float v[2];
#pragma unroll
              for (int h = 0; h < 2; ++h) {
                const float got = __uint_as_float(__shfl_xor_sync(0xffffffffu, low ? r[t + 2 + h] : r[t + h], 16));
                const float own = __uint_as_float(low ? r[t + h] : r[t + 2 + h]);
                v[h] = low ? skinny::siluOf(own) * got : skinny::siluOf(got) * own;
              }
              const float other = __shfl_xor_sync(0xffffffffu, even ? v[1] : v[0], 1);
              const uint32_t w = even ? skinny::pack2(v[0], other) : skinny::pack2(other, v[1]);
              const int token = t + (low ? 0 : 2) + (even ? 0 : 1);
              asm volatile("st.shared.u32 [%0], %1;" ::"r"(buf + uint32_t(token * kPitch + ((lane & 15) >> 1) * 4)), "r"(w) : "memory");
            }
          } else {
            const bool even = (lane & 1) == 0;
#pragma unroll
            for (int t = 0; t < 32; t += 2) {
              const float v0 = __uint_as_float(r[t]), v1 = __uint_as_float(r[t + 1]);
              const float other = __shfl_xor_sync(0xffffffffu, even ? v1 : v0, 1);
              const uint32_t w = even ? skinny::pack2(v0, other) : skinny::pack2(other, v1);
              asm volatile("st.shared.u32 [%0], %1;" ::"r"(buf + uint32_t((t + (even ? 0 : 1)) * kPitch + (lane >> 1) * 4)), "r"(w) : "memory");
            }
          }
          __syncwarp();
          constexpr int kPieces = kOut / 8, kRowsPer = 32 / kPieces;
          const int piece = lane % kPieces, rr = lane / kPieces;
          const bool colOk = n0 + piece * 8 + 8 <= outCols;
#pragma unroll
          for (int i = 0; i < kPieces; ++i) {
            const int row = i * kRowsPer + rr;
            Vec16 v;
            asm volatile("ld.shared.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(v.x[0]), "=r"(v.x[1]), "=r"(v.x[2]), "=r"(v.x[3]) : "r"(buf + uint32_t(row * kPitch + piece * 16)) : "memory");
            if (colOk && c + row < m.count) st16(out + size_t(c + row) * p.ldc + piece * 8, v);
          }
          __syncwarp();                                        // the tile has been read before the next chunk fills it
        };
        uint32_t ra[32], rb[32];
        tc::tmemLoad32(taddr, ra);
#pragma unroll 1
        for (int c = 0; c < m.count; c += 64) {
          tc::tmemLoadWaitFor(ra);
          if (c + 32 < m.count) tc::tmemLoad32(taddr + uint32_t(c + 32), rb);
          drain(ra, c);
          if (c + 32 < m.count) {
            tc::tmemLoadWaitFor(rb);
            if (c + 64 < m.count) tc::tmemLoad32(taddr + uint32_t(c + 64), ra);
            drain(rb, c + 32);
          }
        }
        tc::fenceBeforeThreadSync();
        __syncwarp();
        if (lane == 0) tc::mbarArriveCluster(leaderBars + 8u * (2u * uint32_t(p.stages) + 2u + uint32_t(a)));
      }
    }
  }

  if (*abortWord) __nanosleep(20000);   // let copies already in flight land before shared memory and TMEM go away
  __syncwarp();
  tc::fenceBeforeThreadSync();
  tc::clusterSync();                    // neither CTA frees TMEM the pair's MMA still writes
  if (warp == 1) tc::tmemDeallocPair(tmemBase, kTmemCols);
}

}  // namespace ragged
}  // namespace purlin
