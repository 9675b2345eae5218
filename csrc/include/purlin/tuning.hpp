// Codesign policy: which regime, variant, chunk size and CTA counts a call gets.
//
// The reference hard-codes about 150 constants per architecture and world size
// as compile-time structs (csrc/include/purlin/host/codesign.cuh:28-792) and
// picks a band with if-chains in each host launcher (host/allReduce.cuh:88-308).
// Here the policy is data: a table of (collective, world, size band) -> Policy
// that is filled from a bandwidth sweep on the machine and cached on disk by the
// Python package; the built-in defaults below are only the starting point of
// that sweep and the fallback when no measured table is loaded.
#pragma once
#include <mutex>
#include <vector>

#include "layout.hpp"

namespace purlin {

struct TuningEntry {
  int32_t collective;   // CollectiveType
  int32_t world;
  uint64_t maxBytes;    // band upper bound (inclusive) on the dispatch size
  Policy policy;
};

// Dispatch size of a call, the quantity bands are keyed on: all-reduce = whole payload,
// all-gather = per-rank input, reduce-scatter = per-rank output, all-to-all = per-peer slice,
// V variants = the largest such piece.
inline uint64_t dispatchBytes(const CollectiveSpec& s) {
  switch (s.type) {
    case CollectiveType::allGatherV:
    case CollectiveType::reduceScatterV: { uint64_t m = 0; for (int q = 0; q < s.world; ++q) m = std::max<uint64_t>(m, s.sizes[q]); return m; }
    case CollectiveType::allToAllV: { uint64_t m = 0; for (int q = 0; q < s.world; ++q) m = std::max<uint64_t>(m, std::max(s.sizes[q], s.outSizes[q])); return m; }
    default: return s.bytes;
  }
}

class TuningTable {
 public:
  static TuningTable& global() { static TuningTable t; return t; }
  void clear() { std::lock_guard<std::mutex> g(mu_); entries_.clear(); }
  void add(const TuningEntry& e) {
    std::lock_guard<std::mutex> g(mu_);
    entries_.push_back(e);
    std::stable_sort(entries_.begin(), entries_.end(), [](const TuningEntry& a, const TuningEntry& b) { return a.maxBytes < b.maxBytes; });
  }
  size_t size() const { return entries_.size(); }
  // The band that holds `bytes`; a payload beyond the largest measured band takes that band's policy (what was measured
  // at 256 MiB is a better guess for 1 GiB than the built-in starting point).
  bool lookup(CollectiveType c, int world, uint64_t bytes, Policy& out) const {
    std::lock_guard<std::mutex> g(mu_);
    const TuningEntry* largest = nullptr;
    for (const TuningEntry& e : entries_) {
      if (e.collective != int32_t(c) || e.world != world) continue;
      if (bytes <= e.maxBytes) { out = e.policy; return true; }
      largest = &e;     // entries are sorted by band
    }
    if (largest) { out = largest->policy; return true; }
    return false;
  }
 private:
  mutable std::mutex mu_;
  std::vector<TuningEntry> entries_;
};

// Built-in starting policy for B200 / NVLink 5 (seeded from the reference's Blackwell
// bands, host/codesign.cuh:193-224,331-371,431-478,546-573, then adjusted to this
// datapath: wider grids, because a B200 has 148 SMs and nothing else is running
// during a standalone collective).
inline Policy defaultPolicy(const CollectiveSpec& s, const WorkspaceLayout& ws) {
  Policy p;
  const int W = s.world;
  const uint64_t n = dispatchBytes(s);
  const uint64_t slotPayload = ws.packetStride / 2;
  p.threads = 256;
  p.unroll = 8;
  p.mmDepth = 4;
  p.weighted = 1;
  p.perStreamThreshold = std::min<uint64_t>(256ull << 10, slotPayload);
  const bool nvls = s.multicastAvailable && s.mode == ReductionMode::nonDeterministic;
  auto lrBlocks = [&](uint64_t bytes) { return int(std::min<uint64_t>(std::max<uint64_t>(ceilDiv(bytes, uint64_t(p.threads) * 8), 1), 128)); };
  switch (s.type) {
    case CollectiveType::allReduce: {
      const uint64_t oneShotMax = W <= 2 ? (1ull << 20) : W <= 4 ? (128ull << 10) : (64ull << 10);
      const uint64_t twoShotMax = W <= 2 ? 0 : std::min<uint64_t>(2ull << 20, (slotPayload / 2) * W);
      if (n <= oneShotMax && n <= slotPayload) {
        p.regime = int32_t(Regime::latency); p.arPath = int32_t(AllReducePath::direct);
        p.lrBlocks = lrBlocks(n); p.lrMulticast = nvls ? 1 : 0;
      } else if (n <= twoShotMax && n % (uint64_t(W) * 32) == 0) {
        p.regime = int32_t(Regime::latency); p.arPath = int32_t(AllReducePath::composed);
        p.lrBlocks = lrBlocks(n / W * 2); p.lrMulticast = nvls ? 1 : 0;
      } else {
        p.regime = int32_t(Regime::throughput);
        p.arPath = int32_t(W <= 2 ? AllReducePath::direct : AllReducePath::composed);
        p.memType = int32_t(nvls && W > 2 ? MemType::multimem : MemType::unicast);
        p.threads = 256;
        p.putBlocks = 32; p.consumeBlocks = p.memType == int32_t(MemType::multimem) ? 32 : 48; p.gatherBlocks = 32;
        p.chunkBytes = n <= (4ull << 20) ? 0 : n <= (64ull << 20) ? (2ull << 20) : (8ull << 20);
      }
      break;
    }
    case CollectiveType::allGather:
    case CollectiveType::allGatherV: {
      const uint64_t lrMax = W <= 2 ? (512ull << 10) : W <= 4 ? (256ull << 10) : (64ull << 10);
      if (n <= lrMax && n <= slotPayload) { p.regime = int32_t(Regime::latency); p.lrBlocks = lrBlocks(n * W); }
      else {
        p.regime = int32_t(Regime::throughput); p.putBlocks = 24; p.localBlocks = 8; p.consumeBlocks = 8 * (W - 1) > 64 ? 64 : 8 * (W - 1);
        if (W == 2) p.consumeBlocks = 32;
        p.chunkBytes = n <= (2ull << 20) ? 0 : (2ull << 20);
      }
      break;
    }
    case CollectiveType::reduceScatter:
    case CollectiveType::reduceScatterV: {
      const uint64_t lrMax = W <= 2 ? (512ull << 10) : W <= 4 ? (256ull << 10) : (128ull << 10);
      if (n <= lrMax && n <= slotPayload) { p.regime = int32_t(Regime::latency); p.lrBlocks = lrBlocks(n * W); }
      else {
        p.regime = int32_t(Regime::throughput); p.putBlocks = std::max(32, W); p.consumeBlocks = 48;
        p.chunkBytes = n <= (2ull << 20) ? 0 : (2ull << 20);
      }
      break;
    }
    case CollectiveType::allToAll: {
      const uint64_t lrMax = W <= 4 ? (256ull << 10) : (128ull << 10);
      if (n <= lrMax && n <= slotPayload) { p.regime = int32_t(Regime::latency); p.lrBlocks = lrBlocks(n * W); }
      else {
        p.regime = int32_t(Regime::throughput); p.putBlocks = std::max(4 * (W - 1), 16); p.localBlocks = 8;
        p.consumeBlocks = std::max(8 * (W - 1), 32) > 64 ? 64 : std::max(8 * (W - 1), 32);
        p.chunkBytes = n <= (2ull << 20) ? 0 : (2ull << 20);
      }
      break;
    }
    case CollectiveType::allToAllV: {
      // no whole-collective latency branch: the packet path is chosen per stream inside the plan
      p.regime = int32_t(Regime::throughput); p.putBlocks = std::max(4 * (W - 1), 16); p.localBlocks = 8;
      p.consumeBlocks = std::max(8 * (W - 1), 32) > 64 ? 64 : std::max(8 * (W - 1), 32);
      p.chunkBytes = 1ull << 20;
      break;
    }
  }
  return p;
}

// The fixed-size collective whose measured bands a variable-length call may borrow.
inline bool fixedSibling(CollectiveType t, CollectiveType& out) {
  switch (t) {
    case CollectiveType::allGatherV: out = CollectiveType::allGather; return true;
    case CollectiveType::reduceScatterV: out = CollectiveType::reduceScatter; return true;
    case CollectiveType::allToAllV: out = CollectiveType::allToAll; return true;
    default: return false;
  }
}

inline Policy selectPolicy(const CollectiveSpec& s, const WorkspaceLayout& ws) {
  Policy p;
  const TuningTable& table = TuningTable::global();
  bool found = table.lookup(s.type, s.world, dispatchBytes(s), p);
  if (!found) {
    // No band measured for a variable-length form: borrow the band its fixed-size sibling measured for the largest
    // stream of this call (CTA counts and chunk size carry over; the switch variants were measured for whole, equal
    // slices only and are dropped). A borrowed policy that does not fit the call falls back like any other (planFor).
    CollectiveType sibling;
    if (fixedSibling(s.type, sibling) && table.lookup(sibling, s.world, dispatchBytes(s), p)) {
      const Policy builtIn = defaultPolicy(s, ws);
      if (s.type == CollectiveType::allToAllV && p.regime != int32_t(Regime::throughput)) return builtIn;   // packets are chosen per stream there
      p.memType = int32_t(MemType::unicast);
      p.lrMulticast = 0;
      p.weighted = 1;
      if (p.perStreamThreshold == 0) p.perStreamThreshold = builtIn.perStreamThreshold;
      found = true;
    }
  }
  if (found) {
    // a measured entry may ask for NVLS; drop it where this call cannot use it
    if (!s.multicastAvailable || s.mode == ReductionMode::deterministic) { p.memType = int32_t(MemType::unicast); p.lrMulticast = 0; }
    return p;
  }
  return defaultPolicy(s, ws);
}

// The policy of a collective whose ranks share one GPU: CTAs of one virtual rank among its share of the SMs. Here every role moves its bytes through the same HBM (over NVLink a consumer
// needs far more CTAs than a producer), so the roles share the CTAs by the bytes they read and write; each stream keeps at
// least one. One CTA per stream for everything but the reducers left most of the work to a few CTAs: device time of an all-reduce
// of 64 MiB by 4 ranks 471 -> 365 us, reduce-scatter of 2 x 1 MB 32 -> 12.6 us. What bounds a CTA is the bytes it has in flight, and a
// reducer has half of a copier's (8 x 16 against 8 x 32 bytes a thread), so its bytes count twice: 64 MiB by 4 ranks 352 -> 261 us, reduce-
// scatter 4 x 16 MiB 205 -> 162. Where the streams alone take most CTAs of a rank (8 ranks: 15 of 18), CTAs of 128 threads, two on an SM,
// leave the reducers their part: all-reduce of 64 MiB by 8 ranks 827 -> 485, reduce-scatter 8 x 8 MiB 394 -> 322.
inline void fitEmulated(Policy& p, const CollectiveSpec& s, const WorkspaceLayout& ws, int sms) {
  const int W = s.world;
  // (a bulk ring of seven tiles or more leaves an SM one CTA: measured bands with a ring keep one)
  const bool small = s.op == ConsumeOp::reduce && W > 4 && W <= 8 && p.regime == int32_t(Regime::throughput) && p.stageDepth == 0;
  if (small) p.threads = 128;
  int perRank = std::max((small ? 2 * sms : sms) / W, 2);
  p.lrBlocks = std::min(p.lrBlocks, perRank);
  const bool reduce = s.op == ConsumeOp::reduce, whole = reduce && isPacked(s.in), composed = whole && p.arPath == int32_t(AllReducePath::composed);
  const double w = W;
  // bytes per role, in units of one rank's share: {stage, local, consume or reduce, gather}
  double work[4] = {2, 0, 0, 0};
  int least[4] = {1, 0, 1, 0};
  if (composed) { work[2] = 2 * (1 + 2 / w); work[3] = 2 * (w - 1) / w; least[0] = W; least[3] = W - 1; }
  else if (whole) { work[2] = w + 1; }          // (two ranks, one stream: 64 MiB 155 us like this, 251 with twice the weight)
  else if (reduce) { work[0] = 2 * w; work[2] = 2 * (w + 1); least[0] = W; }
  else if (isScattered(s.in)) { work[0] = 2 * (w - 1); work[1] = 2; work[2] = 2 * (w - 1); least[0] = W - 1; least[1] = 1; least[2] = W - 1; }
  else { work[1] = 2; work[2] = 2 * (w - 1); least[1] = 1; least[2] = W - 1; }
  if (s.type == CollectiveType::allToAllV) { --perRank; work[1] = 0; }   // its short streams get a range of localBlocks CTAs of their own
  int n[4], used = 0;
  for (int i = 0; i < 4; ++i) { n[i] = least[i]; used += n[i]; }
  for (; used < perRank; ++used) {            // one CTA at a time to the role that has most bytes per CTA
    int most = -1;
    for (int i = 0; i < 4; ++i) if (least[i] && (most < 0 || work[i] / n[i] > work[most] / n[most])) most = i;
    ++n[most];
  }
  if (reduce && n[0] > least[0]) {            // the streams are of equal size: CTAs that only some of them would get help the reducers more
    const int uneven = n[0] % least[0];
    n[0] -= uneven; n[2] += uneven;
  }
  // Few and large chunks once there are enough of them: a chunk costs every stream a barrier and a flag. A payload larger than the staging
  // half streams through windows of it, where a large chunk must leave room for others in flight (48 MiB, us, large / as chosen: 4 ranks, one in a window
  // 491 / 331, two 303 / 328; 8 ranks, one 814 / 419, two 503 / 466, three 431 / 437; 3 ranks, two 264 / 273, 5 ranks, four 324 / 382). One that no
  // window holds is cut into quarters of a window by the plan (3 ranks, staging of 4 MiB: 299 / 521).
  const uint64_t large = 4ull << 20, inWindow = roundDown(ws.stagingTRSize / uint64_t(W), uint64_t(kAccessAlign)) / roundUp(large / uint64_t(W), uint64_t(kAccessAlign));
  if (composed && p.chunkBytes && s.bytes >= (12ull << 20) && (s.bytes <= ws.stagingTRSize || inWindow == 0 || inWindow >= (W <= 4 ? 2u : 3u))) p.chunkBytes = std::max<uint64_t>(p.chunkBytes, large);
  p.putBlocks = n[0]; p.localBlocks = std::max(n[1], 1); p.consumeBlocks = n[2]; p.gatherBlocks = std::max(n[3], 1);
}

}  // namespace purlin
