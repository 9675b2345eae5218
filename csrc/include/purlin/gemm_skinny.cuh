// GEMM for few activation rows: C[T, N] = X[T, K] * W[N, K]^T with T up to a few hundred (decode), plain or per expert.
//
// What bounds it is the read of W from HBM (2 * N * K bytes against 2 * T * N * K flops: below about 250 rows the tensor
// cores have time to spare), so the kernel is laid out to keep W streaming from every SM:
//   * W fills the 128 rows of the MMA and the activations are its columns (as many as there are, in steps of 16), so no
//     tensor-core row and no load is spent on padding rows of X;
//   * a tile is 128 rows of W, its k-range is split over a cluster of `split` CTAs. The fp32 partial tiles meet in
//     distributed shared memory and are added in ascending k order: the same bits on every call, no scratch in global
//     memory, no counter, no second launch;
//   * two CTAs per SM (up to 128 columns), each with its own ring of TMA stages: while one drains its accumulator the
//     other one's loads are in flight.
// With `counts` the rows of X are grouped: expert e owns counts[e] consecutive rows and rows [e * N, (e + 1) * N) of W.
// The counts are read on the device, so nobody has to wait for them on the host; an expert without rows reads nothing.
#pragma once
#include <cuda.h>
#include <cuda_bf16.h>

#include "atom.cuh"
#include "gemm_route.hpp"
#include "tc_sm100.cuh"

namespace purlin {
namespace skinny {

constexpr int kThreads = 192;                  // warp 0: TMA, warp 1: MMA, warps 2-5: TMEM -> shared memory; all: the sum

struct alignas(64) Maps { CUtensorMap w, x; };

struct Params {
  int N, K, tokens;        // N: rows of W per expert; tokens: rows of X (with counts: an upper bound of their sum); exchanged with kTokenRows
  int passTokens;          // columns of one pass: multiple of tokenBox
  int columnGroups;        // without counts: this many CTAs share a tile's columns, a pass each (blockIdx.y)
  int tokenBox;            // rows of one X load: 16 or 32
  int stages, tmemCols;
  int ahead;               // k-blocks of W that are asked into L2 while the kernel before this one drains (0 where it has ended, and with counts)
  const int32_t* counts;   // rows per expert, or null: one group of `tokens` rows
  __nv_bfloat16* C;
  int ldc;
  uint32_t* status;        // optional: {code, where, tile, k-block} of the first wait that gave up
  uint64_t timeoutNs;
};

PURLIN_D void recordTimeout(uint32_t* status, uint32_t where, uint32_t a, uint32_t b) {
  if (status && atomicCAS(status, 0u, uint32_t(kStatusTimeoutBarrier)) == 0u) { status[1] = where; status[2] = a; status[3] = b; __threadfence(); }
}

// Rows of a group and sums of them never count past the `limit` rows that there are, whatever the counts say: a count is cut to
// [0, limit] and a sum stays at the limit (neither term is above it, so the unsigned sum cannot wrap).
PURLIN_D uint32_t groupRowsOf(int32_t count, uint32_t limit) { return count > 0 ? min(uint32_t(count), limit) : 0u; }
PURLIN_D uint32_t addRows(uint32_t a, uint32_t b, uint32_t limit) { return min(a + b, limit); }

// (volatile keeps these loads behind the cluster barriers; they may overlap one another and the sums)
PURLIN_D float4 ldCluster4(uint32_t addr) {
  float4 v;
  asm volatile("ld.shared::cluster.v4.f32 {%0,%1,%2,%3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(addr));
  return v;
}
PURLIN_D float ldCluster1(uint32_t addr) {
  float v;
  asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v) : "r"(addr));
  return v;
}
PURLIN_D uint32_t pack2(float lo, float hi) {
  const __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);
  return *reinterpret_cast<const uint32_t*>(&v);
}
PURLIN_D float siluOf(float x) { return __fdividef(x, 1.f + __expf(-x)); }

// eight neighbouring values of one token's partial tiles, added over the cluster in ascending k order
PURLIN_D void sumPartials(const uint32_t (&peer)[kMaxSplit], int split, uint32_t offset, float (&s)[8]) {
#pragma unroll
  for (int e = 0; e < 8; ++e) s[e] = 0.f;
#pragma unroll
  for (int q = 0; q < kMaxSplit; ++q) {
    if (q < split) {
      const float4 a = ldCluster4(peer[q] + offset), b = ldCluster4(peer[q] + offset + 16);
      s[0] += a.x; s[1] += a.y; s[2] += a.z; s[3] += a.w;
      s[4] += b.x; s[5] += b.y; s[6] += b.z; s[7] += b.w;
    }
  }
}

// the same value of eight neighbouring columns (tokens) of the partial tiles
PURLIN_D void sumPartialColumns(const uint32_t (&peer)[kMaxSplit], int split, uint32_t offset, float (&s)[8]) {
#pragma unroll
  for (int e = 0; e < 8; ++e) s[e] = 0.f;
#pragma unroll
  for (int q = 0; q < kMaxSplit; ++q) {
    if (q < split) {
#pragma unroll
      for (int e = 0; e < 8; ++e) s[e] += ldCluster1(peer[q] + offset + uint32_t(e * kRows * 4));
    }
  }
}

// kWeightRows: the MMA's rows are rows of W and its columns are tokens, as described above. kTokenRows: the same kernel with
// the operands' roles exchanged, for few rows of W (a router) against many tokens: `w` then maps X, `x` maps W, and a row of
// the partial tile is a row of C.
enum { kWeightRows = 0, kWeightRowsSwiglu = 1, kTokenRows = 2 };

template <int MODE>
__global__ void __launch_bounds__(kThreads, 2) skinnyGemmKernel(const __grid_constant__ Maps maps, const __grid_constant__ Params p) {
  extern __shared__ unsigned char smemRaw[];
  const uint32_t rawAddr = tc::smemAddr(smemRaw);
  const uint32_t base = (rawAddr + 1023u) & ~1023u;           // swizzled tiles need 1024-byte alignment
  unsigned char* smem = smemRaw + (base - rawAddr);
  const int xBytes = p.passTokens * kK * 2;
  const uint32_t stageBytes = uint32_t(kWBytes + xBytes);     // a multiple of 2 KiB: [W][X]
  const uint32_t barBase = base + uint32_t(p.stages) * stageBytes;
  auto fullBar = [&](uint32_t s) { return barBase + 8u * s; };
  auto emptyBar = [&](uint32_t s) { return barBase + 8u * (uint32_t(p.stages) + s); };
  const uint32_t accFull = barBase + 8u * (2u * uint32_t(p.stages)), mmasDone = accFull + 8u;
  uint32_t* words = reinterpret_cast<uint32_t*>(smem + size_t(p.stages) * stageBytes + 8 * (2 * p.stages + 2));
  volatile uint32_t* tmemBaseWord = words;
  volatile int* abortWord = reinterpret_cast<volatile int*>(words + 1);
  volatile int* groupRows = reinterpret_cast<volatile int*>(words + 2);   // first row and number of rows of this expert

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  uint32_t split;
  asm volatile("mov.u32 %0, %%cluster_nctaid.x;" : "=r"(split));
  const uint32_t part = tc::clusterCtaRank();
  const int tile = int(blockIdx.x / split), expert = p.counts ? int(blockIdx.y) : 0;

  if (threadIdx.x == 0) {
    for (int s = 0; s < p.stages; ++s) { tc::mbarInit(fullBar(s), 1); tc::mbarInit(emptyBar(s), 1); }
    tc::mbarInit(accFull, 1);
    tc::mbarInit(mmasDone, 1);
    *abortWord = 0;
    tc::mbarFenceInit();
    tc::tmaPrefetchDescriptor(&maps.w);
    tc::tmaPrefetchDescriptor(&maps.x);
  }
  const int kBlocks = (p.K + kK - 1) / kK;
  const int kBegin = int(int64_t(kBlocks) * part / split), kEnd = int(int64_t(kBlocks) * (part + 1) / split);
  // The first lap of the ring is asked into L2 while the kernel before this one drains (a hint: nothing of it is read before the wait, so
  // W may be what that kernel writes). 1 x 8192 x 3584 MLP block 36.0 -> 34.1 us, 32 x 8192 x 8192 74.0 -> 71.8; half a lap gains less,
  // two or the whole range take bandwidth from the kernel that still runs (35.7, 39.1 us).
  if (warp == 0 && lane == 0)
    for (int kb = kBegin; kb < min(kEnd, kBegin + p.ahead); ++kb) tc::tmaPrefetchL2(&maps.w, kb * kK, expert * p.N + tile * kRows);
  if (warp == 1) { tc::tmemAlloc(tc::smemAddr(words), uint32_t(p.tmemCols)); tc::tmemRelinquish(); }
  tc::gridDependencyWait();                                   // from here on memory that earlier kernels write may be read
  if (warp == 2) {
    const uint32_t limit = uint32_t(p.tokens);
    uint32_t first = 0, rows = limit;
    if (p.columnGroups > 1) {
      first = min(blockIdx.y * uint32_t(p.passTokens), limit);
      rows = min(uint32_t(p.passTokens), limit - first);
    }
    if (p.counts) {
      for (int e = lane; e < expert; e += 32) first = addRows(first, groupRowsOf(p.counts[e], limit), limit);
#pragma unroll
      for (int o = 16; o; o >>= 1) first = addRows(first, __shfl_xor_sync(0xffffffffu, first, o), limit);
      rows = min(groupRowsOf(p.counts[expert], limit), limit - first);
    }
    if (lane == 0) { groupRows[0] = int(first); groupRows[1] = int(rows); }
  }
  tc::fenceBeforeThreadSync();
  __syncthreads();
  tc::fenceAfterThreadSync();
  const uint32_t tmemBase = *tmemBaseWord;
  const int firstRow = groupRows[0], rows = groupRows[1];
  uint32_t peer[kMaxSplit];                                   // every CTA's partial tile [token][128] fp32, over the stages' memory
#pragma unroll
  for (int q = 0; q < kMaxSplit; ++q) peer[q] = uint32_t(q) < split ? tc::mapToCta(base, uint32_t(q)) : 0u;

  uint32_t st = 0, ph = 0;                                    // ring position and phase of the producer / the MMA issuer
  bool ok = true;
  int pass = 0;
  for (int t0 = 0; t0 < rows; t0 += p.passTokens, ++pass) {
    const int count = min(p.passTokens, rows - t0);
    const int loads = (count + p.tokenBox - 1) / p.tokenBox;
    const int cols = loads * p.tokenBox;                      // columns of the MMA; those past `count` are never stored
    if (warp == 0) {
      if (lane == 0) {
        const int wRow = expert * p.N + tile * kRows;
        for (int kb = kBegin; kb < kEnd && ok; ++kb) {
          ok = tc::mbarWait(emptyBar(st), ph ^ 1, abortWord, p.timeoutNs);
          if (!ok) { recordTimeout(p.status, 1, tile, kb); break; }
          const uint32_t sW = base + st * stageBytes, sX = sW + kWBytes;
          tc::mbarExpectTx(fullBar(st), uint32_t(kWBytes + cols * kK * 2));
          tc::tmaLoad2d(sW, &maps.w, kb * kK, wRow, fullBar(st));
          for (int i = 0; i < loads; ++i)
            tc::tmaLoad2d(sX + uint32_t(i * p.tokenBox * kK * 2), &maps.x, kb * kK, firstRow + t0 + i * p.tokenBox, fullBar(st));
          if (++st == uint32_t(p.stages)) { st = 0; ph ^= 1; }
        }
      }
    } else if (warp == 1) {
      if (lane == 0) {
        const uint32_t idesc = tc::instrDescBf16(uint32_t(cols), uint32_t(kRows));
        const uint64_t descW = tc::smemDescSw128(base), descX = tc::smemDescSw128(base + kWBytes);
        for (int kb = kBegin; kb < kEnd && ok; ++kb) {
          ok = tc::mbarWait(fullBar(st), ph, abortWord, p.timeoutNs);
          if (!ok) { recordTimeout(p.status, 3, tile, kb); break; }
          tc::fenceAfterThreadSync();
          const uint64_t step = uint64_t(st * (stageBytes >> 4));
#pragma unroll
          for (int k = 0; k < kK / 16; ++k)
            tc::mma(tmemBase, descW + step + 2 * k, descX + step + 2 * k, idesc, uint32_t(kb != kBegin || k != 0));
          tc::mmaCommit(emptyBar(st));
          if (++st == uint32_t(p.stages)) { st = 0; ph ^= 1; }
        }
        if (ok) tc::mmaCommit(accFull);
      }
    } else {
      // ---- this CTA's partial tile: TMEM (lane = row of W, column = token) -> shared memory [token][row of W] ----
      const int quarter = warp & 3;                           // a warp may only touch TMEM lanes [32 * (warp % 4), +32)
      ok = tc::mbarWait(accFull, uint32_t(pass & 1), abortWord, p.timeoutNs);
      ok = __all_sync(0xffffffffu, ok);
      if (!ok && lane == 0) recordTimeout(p.status, 5, tile, pass);
      if (ok) {
        // every load of the pass has landed and every MMA has read its stage, so the stages' memory is free
        tc::fenceAfterThreadSync();
        const uint32_t taddr = tmemBase + (uint32_t(quarter * 32) << 16);
        float* mine = reinterpret_cast<float*>(smem) + quarter * 32 + lane;
        for (int c = 0; c < count; c += 32) {
          uint32_t r[32];
          tc::tmemLoad32(taddr + uint32_t(c), r);             // reads up to 16 columns past `cols`: allocated, not used
          tc::tmemLoadWaitFor(r);
#pragma unroll
          for (int i = 0; i < 32; ++i) if (c + i < count) mine[size_t(c + i) * kRows] = __uint_as_float(r[i]);
        }
        tc::fenceBeforeThreadSync();
      }
    }
    // A wait that gave up is everybody's business: the partial tile of this CTA is not what its peers would add. They learn of it
    // through their own abort words, written before the cluster barrier after which they are read.
    if (!ok) {
      const uint32_t word = tc::smemAddr(words + 1);
      for (uint32_t q = 0; q < split; ++q) asm volatile("st.shared::cluster.u32 [%0], %1;" ::"r"(tc::mapToCta(word, q)), "r"(1) : "memory");
    }
    __syncwarp();
    tc::clusterSync();                                        // every partial tile of the cluster is in shared memory
    // Only now may the next kernel take the free places: earlier, its CTAs would crowd the SMs that this one leaves empty.
    tc::gridLaunchDependents();
    // ---- the sum: CTA `part` finishes its share of the tokens, 8 output columns per thread ----
    if (MODE == kTokenRows && *abortWord == 0) {
      // row r of the tile, 8 of its columns per thread; neighbouring lanes read neighbouring rows
      const int begin = kRows * int(part) / int(split), mine = kRows * int(part + 1) / int(split) - begin, pieces = (count + 7) / 8;
      for (int i = int(threadIdx.x); i < mine * pieces; i += kThreads) {
        const int r = begin + i % mine, piece = i / mine, row = tile * kRows + r;
        if (row >= p.N) continue;
        float v[8];
        sumPartialColumns(peer, int(split), uint32_t(piece * 8 * kRows + r) * 4u, v);
        st16(p.C + size_t(row) * p.ldc + firstRow + t0 + piece * 8, Vec16{{pack2(v[0], v[1]), pack2(v[2], v[3]), pack2(v[4], v[5]), pack2(v[6], v[7])}});
      }
    } else if (*abortWord == 0) {
      constexpr bool SWIGLU = MODE == kWeightRowsSwiglu;
      constexpr int kOut = SWIGLU ? kRows / 2 : kRows, kPieces = kOut / 8;
      const int outCols = SWIGLU ? p.N / 2 : p.N, n0 = tile * kOut;
      const int begin = int(int64_t(count) * part / split) * kPieces, end = int(int64_t(count) * (part + 1) / split) * kPieces;
#pragma unroll 2
      for (int i = begin + int(threadIdx.x); i < end; i += kThreads) {
        const int t = i / kPieces, piece = i % kPieces;
        if (n0 + piece * 8 + 8 > outCols) continue;
        float v[8];
        if constexpr (SWIGLU) {
          // rows alternate 16 of gate and 16 of up
          const uint32_t at = uint32_t(t * kRows + (piece >> 1) * 32 + (piece & 1) * 8) * 4u;
          float u[8];
          sumPartials(peer, int(split), at, v);
          sumPartials(peer, int(split), at + 64u, u);
#pragma unroll
          for (int e = 0; e < 8; ++e) v[e] = siluOf(v[e]) * u[e];
        } else {
          sumPartials(peer, int(split), uint32_t(t * kRows + piece * 8) * 4u, v);
        }
        st16(p.C + size_t(firstRow + t0 + t) * p.ldc + n0 + piece * 8, Vec16{{pack2(v[0], v[1]), pack2(v[2], v[3]), pack2(v[4], v[5]), pack2(v[6], v[7])}});
      }
    }
    // Nobody overwrites or leaves behind a partial tile that a peer still reads; the next pass's TMA writes into that
    // memory come after these generic-proxy accesses.
    tc::fenceProxyAsync();
    tc::clusterSync();
  }
  if (*abortWord) {
    // copies and MMAs under way end before shared memory and TMEM go away: the last copy into each stage (of this lap of the ring
    // or the one before; a stage never used counts as landed), the last MMA issued
    if (warp == 0 && lane == 0) for (uint32_t s = 0; s < uint32_t(p.stages); ++s) tc::mbarDrain(fullBar(s), s < st ? ph : ph ^ 1);
    if (warp == 1 && lane == 0) { tc::mmaCommit(mmasDone); tc::mbarDrain(mmasDone, 0); }
    __syncwarp();
  }
  tc::fenceBeforeThreadSync();
  __syncthreads();
  if (warp == 1) tc::tmemDealloc(tmemBase, uint32_t(p.tmemCols));
}

}  // namespace skinny
}  // namespace purlin
