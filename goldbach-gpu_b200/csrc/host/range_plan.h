// range_plan.h -- how a range call is cut and which kernels it takes (plain C++,
// no CUDA: also compiled by the host tests).
#pragma once
#include <algorithm>
#include <cmath>
#include <cstdint>

namespace gb {

// Chunk width when the caller leaves it open: the one with the least time on
// the fullest SM, for pieces cut into chunks each by itself (`pieces` of `len`
// n and one of `tail`).  A chunk costs ne + fixed, in n; an SM runs two CTAs at
// once, and one alone takes 0.77 of a pair's time.  For a few numbers of chunks
// per SM the narrowest width that needs no more is tried, in steps of 512 n.
// Powers of two left a last wave of a few chunks: 2e8 n near 1e12 329 -> 257
// us, 5e8 n near 1e9 469 -> 396, 4e7 n near 1e15 (masked) 237 -> 189.  With an odd
// number of five or more chunks of the widest per SM, the widest is kept: the last
// chunk overlaps the uneven ends of the others, and narrower ones mostly add their
// fixed cost.  Kernel us at the widest / narrower, in segments of 2^27 n: near 1e10
// 6.5e8 n 574 / 539, 7.5e8 580 / 617, 1.05e9 799 / 884, 1.3e9 1024 / 990, 1.6e9 1250 /
// 1179; near 1e12 756 / 727, 766 / 828, 1047 / 1185, 1346 / 1332, 1647 / 1581; masked
// near 1e15 the same within 1%; with per-n output near 1e9 4.1e7 n 190 / 170, 4.7e7
// 193 / 196, 6e7 248 / 226, 8.5e7 317 / 320.  (So it loses where few of the SMs have
// the odd chunk, up to 10%, and gains up to 12% where most have.)
// No width passes the longest piece: it would cut nothing, and the chunk's own
// sieving primes and shared memory follow it.
inline uint32_t balanced_chunk(uint64_t pieces, uint64_t len, uint64_t tail, double fixed, int sm_count, uint32_t least,
                               uint32_t most) {
  const uint64_t longest = pieces ? std::max(len, tail) : tail;
  if (longest < most) most = std::max<uint32_t>(least, ((uint32_t)longest + 511) & ~511u);
  auto chunks = [&](uint64_t ne) { return pieces * ((len + ne - 1) / ne) + (tail + ne - 1) / ne; };
  const double total = (double)pieces * (double)len + (double)tail;
  double best = -1;
  uint32_t pick = most;
  const uint64_t at_most = (chunks(most) + sm_count - 1) / sm_count;  // chunks per SM at the widest
  if (at_most >= 5 && (at_most & 1)) return most;
  for (uint64_t k = std::max<uint64_t>(1, at_most); k <= at_most + 5; ++k) {
    // the narrowest width (a multiple of 512) with at most k sm_count chunks
    uint64_t lo = std::max<uint64_t>(least, (uint64_t)(total / (double)(k * sm_count)) & ~511ull), hi = most;
    if (chunks(hi) > k * sm_count) continue;
    if (lo > hi) lo = hi;
    lo = (lo + 511) & ~511ull;
    while (lo < hi) {
      const uint64_t mid = (lo + hi) / 1024 * 512;
      if (chunks(mid) <= k * sm_count) hi = mid;
      else lo = mid + 512;
    }
    const double t = ((double)hi + fixed) * (0.5 * (double)k + (k & 1 ? 0.27 : 0.0));
    if (best < 0 || t < best) {
      best = t;
      pick = (uint32_t)hi;
    }
    if (hi <= least) break;
  }
  return pick;
}

// Whether a range of `count` n from `start` on, in `pieces` segments that form
// `runs` stretches without a gap (a shard's share of `segments`), goes through
// masks of the large-prime pass (range_masked); root: its largest sieving prime;
// ne: the width of its chunks without them.  A chunk spends 0.6 ns on each of its
// sieving primes, whatever its width, and with two CTAs per SM a wave of chunks
// as much; the masks leave it the primes up to 2^16.  They cost, in ns: 25000 and
// 0.05 a prime for the pass, 1.5 per n for its marks, 14000 per further wave (a
// chunk's window is looked up and its masks read), 400 per run (each prime walks
// all of them in a row), and 10 per piece on the host.  Chunks alone against
// masks, us per call: 1e6 n near 1e11 115 / 116, 1e12 132 / 126, 1e13 207 / 126; 1e7
// n near 1e12 144 / 153, 4e12 185 / 157; 3e7 near 4e12 207 / 208; 1e7 near 1e12 in
// segments of 1000 n 2379 / 1496, every second of them 1241 / 3059, of 30000 n 157 /
// 199, near 1e13 243 / 212.  From kMaskedWidth n per SM on the chunks are wide,
// their own cost is below the marks', and the line lies at kMaskedRoot whatever
// the count: 1e9 n near 1e13 1.46 / 2.11 ms, 5e13 2.04 / 1.91, 3e14 3.96 / 2.07, near
// 1e17 67 / 3.2.
// The range must start beyond every sieving prime, and the pass's quotient
// estimates need p > g0 / 2^42 (masked_bound).
constexpr uint64_t kRangeMaskEvens = 1ull << 28;   // of a run, and of the masks made at a time
constexpr uint64_t kRangeMaskPieces = 1ull << 20;
constexpr uint64_t kMaskedWidth = 1ull << 18, kMaskedRoot = 6000000;

inline bool range_masked_pays(int sm_count, uint64_t start, uint64_t count, uint64_t root, uint64_t pieces,
                              uint64_t runs, uint32_t ne, uint64_t segments) {
  if (start < (8ull << 30) || root < (1ull << 16)) return false;
  if (segments > 0xffffffffull) return false;  // (a piece's index takes 32 bits)
  if (pieces + count / kRangeMaskEvens > kRangeMaskPieces) return false;  // (some 500 bytes of descriptors each)
  if (root >= kMaskedRoot) return true;
  if (count >= kMaskedWidth * (uint64_t)sm_count) return false;
  const double primes = 1.1 * (double)root / std::log((double)root) - 6542;  // beyond 2^16
  const double waves = std::max(1.0, std::max((double)pieces, (double)count / ne) / (2.0 * sm_count));
  const double cost = 25e3 + 0.05 * primes + 1.5e-3 * (double)count + 14e3 * (waves - 1) + 400.0 * (double)runs +
                      10.0 * (double)pieces;
  return cost < 0.6 * primes * waves;
}

}  // namespace gb
