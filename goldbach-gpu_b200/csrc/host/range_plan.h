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
// us, 5e8 n near 1e9 469 -> 396, 4e7 n near 1e15 (masked) 237 -> 189.  With five or
// more chunks of the widest per SM, an odd number, the last one overlaps the
// uneven ends of the others and narrower chunks only add their fixed cost:
// 6e8 and 1e9 n near 1e12 689 and 1045 us at the widest, 717 and 1105 narrower.
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

}  // namespace gb
