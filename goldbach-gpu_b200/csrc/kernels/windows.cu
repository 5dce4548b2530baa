// windows.cu -- batched verification of many independent windows of even n:
// the large-prime pass, the tested windows, and the expansion of narrow windows
// for the single-n kernel.
//
// The reference verifies one contiguous range at a time with a host loop of
// launches per segment (src/goldbach.cu:420-485).  Windows far out (starts
// up to 1e18) need sieving primes up to 1e9, and every one of those primes
// needs its first multiple in every window: about 1e11 (prime, window)
// pairs for the 4096 seeded windows in [1e15, 1e18], of which only a few
// percent have a multiple in the window at all.  The batch is therefore
// split by prime size:
//   1. this pass: one thread per prime p above the chunk sieve's bound walks
//      the windows (sorted by their top, so only those with p^2 <= top are
//      visited) and clears p's multiples in each window's two class masks
//      (mod-6 layout, bit t <-> q = 6(g0 + t) + c, c in {1, 5}) with global
//      atomicAnd;
//      (narrow windows have their masks made by primality tests instead,
//      see below);
//   2. range6_kernel in windows mode: every (window, chunk) item sieves its
//      q-window in shared memory with the wheel and the primes up to the
//      bound, ANDs in the window's masks, and runs the levelled search;
//   3. the device Phase 2 (range.cu fallback_kernel) for minimal p beyond
//      the halo.
//
// Cost of a pair.  The first mark of class c is t_c = (a_c - g0) mod p, a_1 =
// -1/6 and a_5 = -5/6 (mod p).  One fused multiply-add of g0 (as a double) by
// 1/p onto 1.5 * 2^52 rounds g0 / p to an integer m with an error below 1/4 beside the
// rounding (g0 / p < 2^42, near_inv), held in the double's low bits, and d = m p - g0
// (mod 2^32) is within 3p/4 of zero.  The a_c taken next to zero are within p/6 of it (6
// divides p - 1 or p + 1), so d + a_c lies in (-p, p), and t_c = min(d + a_c, d +
// a_c + p) as unsigned 32-bit numbers when p < 2^31; for larger p a sum below
// zero leaves t_c >= p/12 > 2^27, beyond every mask taken here (< 2^27 bits),
// and d + a_c itself is compared.  So a pair costs one 16-byte load, one FMA,
// one multiply-add, two additions, two add-and-minimum, a minimum and a
// comparison.  (One residue mod p for both classes, the distance from 6 g0 to
// p's next multiple, costs half of that but hits three times as often, and the
// hits are what a wide window pays for: it measured 56 ms against 28.)  The pass
// marks every multiple of p in the window, those below p^2 included (they are
// composite); only p itself must stay, and it can lie in a window only when the
// window starts below 2^32, so those windows (g0 < 2^30) take an exact path with
// the p^2 rule, and so do masks of 2^27 bits or more.
#include <cuda_runtime.h>

#include <cstdint>

#include "../gb_device.cuh"
#include "../gb_internal.h"
#include "gb/gb.h"
#include "prp64.cuh"
#include "sieve6.cuh"

namespace gb {

constexpr int kWinLargeThreads = 256;

// Exact marks of p in window w: first marks from the signed base with the
// p^2 rule (sieve6.cuh), then every p-th bit of both class masks.
__device__ __noinline__ void win_mark_exact(const WinLargeArgs& a, uint32_t w, uint32_t p, uint32_t k) {
  const WinDesc6 d = a.win[w];
  const uint32_t lbits = d.lwords * 32;
  uint32_t t1, t5;
  first_marks6(d.g0, p, __ldg(a.a15 + k), base_mod(d.g0, p, __ldg(a.magic + k)), lbits, t1, t5);
  uint32_t* L1 = a.lmask + d.lbase;
  uint32_t* L5 = L1 + d.lwords;
  for (uint64_t i = t1; i < lbits; i += p) atomicAnd(&L1[i >> 5], ~(1u << (i & 31)));
  for (uint64_t i = t5; i < lbits; i += p) atomicAnd(&L5[i >> 5], ~(1u << (i & 31)));
}

// First window w in [lo, hi) whose top reaches p^2 (windows sorted by q_top).
__device__ __forceinline__ uint32_t first_window(const WinLargeArgs& a, uint64_t pp, uint32_t lo, uint32_t hi) {
  while (lo < hi) {
    const uint32_t mid = (lo + hi) >> 1;
    if (a.win[mid].q_top < pp) lo = mid + 1;
    else hi = mid;
  }
  return lo;
}

// Marks p's multiples in window w from the first marks t1, t5 on, in ascending
// order over both classes: most hits are one mark of either class, so a warp's
// lanes make it together.
__device__ __forceinline__ void win_mark_from(const WinLargeArgs& a, uint32_t w, uint32_t p, uint32_t t1,
                                              uint32_t t5, uint32_t lbits) {
  const WinDesc6& d = a.win[w];
  uint32_t* L = a.lmask + d.lbase;
  const uint32_t lwords = d.lwords;
  for (;;) {
    const bool c1 = t1 <= t5;
    const uint32_t t = c1 ? t1 : t5;
    if (t >= lbits) break;
    atomicAnd(L + (t >> 5) + (c1 ? 0 : lwords), ~(1u << (t & 31)));
    const uint32_t next = lbits - t <= p ? lbits : t + p;
    if (c1) t1 = next;
    else t5 = next;
  }
}

// 1/p to a relative error of 2^-46: the single-precision reciprocal (2^-24 for its
// own rounding and 2^-24 for p's to a float) and one Newton step in double
// precision, which squares it.  With g0 / p < 2^42 (p > 2^20 for the windows,
// masked_bound for ranges) the quotient estimate is then within 2^-4 of exact, and
// g0's rounding to a double adds 2^-11.  A correctly rounded division costs several
// times more and is paid once per prime, which dominates when few windows share
// the pass.
__device__ __forceinline__ double near_inv(uint32_t p) {
  const double pd = (double)p;
  const double r0 = (double)__frcp_rn((float)p);
  return fma(r0, fma(-pd, r0, 1.0), r0);
}

// A warp takes 32 consecutive primes, one per lane, through the windows whose
// top reaches their squares.  A lane keeps its hits in a column of its own in
// shared memory (two predicated instructions a pair, no vote), and the warp
// marks them row by row when a column is nearly full: marking each hit at once
// runs the marking code for one or two lanes at nearly every pair of a wide
// window.  944 windows of 6e6 n on average near 1e18, 3.0e10 pairs and 1.6e9
// marks: 27.6 ms; marking at once 86 ms; at once over all windows in one launch
// (marks missing L2) 57 ms.  What is left is issue: 77% of the slots, about 24
// instructions a pair, 10 of them arithmetic.  The host launches the pass for
// groups of windows whose masks stay in L2 (kLargeGroupBytes): a launch over all
// of them marks a mask of 0.5 GB at random, and every mark reads and writes a
// sector of HBM.
constexpr int kHitRows = 12;  // 48 KB a CTA, 4 CTAs per SM
struct HitQueue {
  uint4 e[kHitRows][32];  // t1, t5, window, prime index
};

// A lane's prime and what a pair needs of it.
struct LargePrime {
  uint32_t k, p, a1, a1p, a5, a5p, lo;
  double inv;
};

constexpr int kPrimesPerLane = 2;  // sharing each window record's load (1: 30.1, 2: 27.6 ms)

__global__ void __launch_bounds__(kWinLargeThreads) win_large_kernel(const __grid_constant__ WinLargeArgs a) {
  constexpr uint32_t kAll = 0xffffffffu;
  constexpr int P = kPrimesPerLane;
  __shared__ HitQueue s_queue[kWinLargeThreads / 32];
  const uint32_t lane = threadIdx.x & 31;
  uint4* const q0 = &s_queue[threadIdx.x >> 5].e[0][lane];
  uint4* q = q0;  // the lane's next row
  auto flush = [&]() {
    const int n = (int)(q - q0) / 32;
    const int rows = (int)__reduce_max_sync(kAll, (uint32_t)n);
    for (int i = 0; i < rows; ++i) {
      if (i >= n) continue;
      const uint4 e = q0[32 * i];
      const uint32_t lbits = a.wl[e.z].lbits, p = __ldg(a.primes + e.w);
      if (lbits == kLargeExact) win_mark_exact(a, e.z, p, e.w);
      else win_mark_from(a, e.z, p, e.x, e.y, lbits);
    }
    q = q0;
    __syncwarp();
  };
  auto pair = [&](const WinLarge& r, const LargePrime& c, uint32_t w, bool visits) {
    const uint32_t m = (uint32_t)__double_as_longlong(fma(r.gd, c.inv, 6755399441055744.0));  // + 1.5 * 2^52
    const uint32_t d = m * c.p + r.ngl;
    const uint32_t t1 = min(d + c.a1, d + c.a1p), t5 = min(d + c.a5, d + c.a5p);
    if (min(t1, t5) < r.lbits && visits) {
      *q = make_uint4(t1, t5, w, c.k);
      q += 32;
    }
  };
  unsigned long long pairs = 0;
  const uint64_t stride = (uint64_t)gridDim.x * kWinLargeThreads * P;
  const uint64_t top0 = a.w_hi > a.w_lo ? a.win[a.w_lo].q_top : 0;
  const uint64_t first = a.k0 + ((uint64_t)blockIdx.x * kWinLargeThreads + (threadIdx.x & ~31u)) * P;
  for (uint64_t kb = first; kb < a.k1; kb += stride) {
    LargePrime c[P];
    uint32_t lo = a.w_hi, hi = 0;
#pragma unroll
    for (int j = 0; j < P; ++j) {
      const uint64_t kk = kb + 32 * j + lane;
      const bool in = kk < a.k1;
      c[j].k = in ? (uint32_t)kk : a.k1 - 1;
      const uint32_t p = c[j].p = __ldg(a.primes + c[j].k);
      const uint64_t pp = (uint64_t)p * p;
      c[j].lo = !in ? a.w_hi : pp <= top0 ? a.w_lo : first_window(a, pp, a.w_lo, a.w_hi);
      pairs += a.w_hi - c[j].lo;
      lo = min(lo, c[j].lo);
      hi = max(hi, c[j].lo);
      c[j].inv = near_inv(p);
      // a_1, a_5 next to zero: (p - 1) / 6 and -(p + 5) / 6 for p = 1 (mod 6),
      // -(p + 1) / 6 and (p - 5) / 6 for p = 5 (mod 6)
      const uint32_t p6 = __umulhi(p, 0xAAAAAAABu) >> 2;  // floor(p / 6)
      const bool one = p - 6 * p6 == 1;
      c[j].a1 = one ? p6 : 0u - p6 - 1;
      c[j].a5 = one ? 0u - p6 - 1 : p6;
      const uint32_t padd = p < 0x80000000u ? p : 0;
      c[j].a1p = c[j].a1 + padd;
      c[j].a5p = c[j].a5 + padd;
    }
    const uint32_t wlo = __reduce_min_sync(kAll, lo), whi = __reduce_max_sync(kAll, hi);
    if (wlo >= a.w_hi) break;  // no window reaches these primes' squares, nor later ones'
    uint4* const near_full = q0 + 32 * (kHitRows - 4 * P);
    uint32_t w = wlo;
    for (; w < whi; ++w) {  // windows that only some of the lanes' primes visit
      if (__any_sync(kAll, q > near_full)) flush();
      const WinLarge r = a.wl[w];
#pragma unroll
      for (int j = 0; j < P; ++j) pair(r, c[j], w, w >= c[j].lo);
    }
#pragma unroll 1
    for (; w + 4 <= a.w_hi; w += 4) {
      if (__any_sync(kAll, q > near_full)) flush();
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const WinLarge r = a.wl[w + i];
#pragma unroll
        for (int j = 0; j < P; ++j) pair(r, c[j], w + i, true);
      }
    }
    for (; w < a.w_hi; ++w) {
      if (__any_sync(kAll, q > near_full)) flush();
      const WinLarge r = a.wl[w];
#pragma unroll
      for (int j = 0; j < P; ++j) pair(r, c[j], w, true);
    }
  }
  flush();
  for (int o = 16; o; o >>= 1) pairs += __shfl_down_sync(kAll, pairs, o);
  if (lane == 0 && pairs) atomicAdd(a.pairs, pairs);
}

cudaError_t launch_win_large(const WinLargeArgs& a, int grid, cudaStream_t s) {
  win_large_kernel<<<grid, kWinLargeThreads, 0, s>>>(a);
  return cudaGetLastError();
}

// ---------------------------------------------------------------------------
// Tested windows.  A window of W even n costs the large-prime pass one pair per
// sieving prime, however narrow it is: 5e7 pairs near 1e18 (about 40 us of the
// GPU at first, 25 now), of which nearly all miss.  Its 2W / ln(top) primes can be had for less
// when it is narrow: sieve with the primes up to a few times its width, which
// leaves about 1.7 times as many q as there are primes, and test those
// (prp64.cuh).  The tests cost about 16 ps per even n near 1e18, so the line
// between the two lies near 1.5e6 n there (gb_windows.cpp, kTestDivisor).
// 4096 windows at offsets in [1e15, 1e18], widths log-uniform in [2^10, 2^24]:
// 145 -> 86 ms in all, of which the presieve 3.3, the tests 13.7 ms; 61 windows
// of at most 2^18 n 6.5 -> 1.9 ms.
constexpr int kPresieveThreads = 512;

// One tile of one window per step: both classes sieved in shared memory, the
// bits past the window's last n cleared, and written to the window's masks.
__global__ void __launch_bounds__(kPresieveThreads, kPresieveCtasPerSm)
    win_presieve_kernel(const __grid_constant__ WinTestArgs a) {
  extern __shared__ uint32_t sm_presieve[];
  uint32_t* pat6 = sm_presieve;
  uint32_t* Q1 = pat6 + kWheel6Words;
  uint32_t* Q5 = Q1 + a.tile_words;
  if (blockIdx.x >= a.tiles) return;
  for (uint32_t i = threadIdx.x; i < kWheel6Words; i += kPresieveThreads) pat6[i] = a.wheel6[i];
  __syncthreads();
  for (uint64_t item = blockIdx.x; item < a.tiles; item += gridDim.x) {
    const uint32_t w = find_item_window(a.tile_off, a.nwin, item);
    const WinDesc6 d = a.win[w];
    const uint32_t wo = (uint32_t)(item - a.tile_off[w]) * a.tile_words;
    const uint32_t nw = min(a.tile_words, d.lwords - wo);
    const int64_t G0 = d.g0 + 32 * (int64_t)wo;
    sieve_window6<kPresieveThreads, true>(Q1, Q5, nw, 32 * nw, G0, d.q_top, pat6, a.primes, a.magic, a.a15,
                                    a.nsieve[nw > 1 ? 32 - __clz(nw - 1) : 0], a.kcoop);
    uint32_t* L = a.lmask + d.lbase + wo;
    for (uint32_t i = threadIdx.x; i < 2 * nw; i += kPresieveThreads) {
      const bool c5 = i >= nw;
      const uint32_t t = c5 ? i - nw : i;
      // bits left in this word with 6(G0 + t) + c <= q_top
      const int64_t keep = (int64_t)((d.q_top - (c5 ? 5 : 1)) / 6) - G0 - 32 * (int64_t)t;
      const uint32_t m = keep < 0 ? 0u : keep >= 31 ? 0xffffffffu : (2u << keep) - 1;
      L[c5 ? d.lwords + t : t] = (c5 ? Q5 : Q1)[t] & m;
    }
    __syncthreads();
  }
}

cudaError_t launch_win_presieve(const WinTestArgs& a, int grid, cudaStream_t s) {
  const size_t smem = (kWheel6Words + 2 * (size_t)a.tile_words) * sizeof(uint32_t);
  win_presieve_kernel<<<grid, kPresieveThreads, smem, s>>>(a);
  return cudaGetLastError();
}

// The q that the masks hold, 32 at a time per warp: a lane takes a mask word
// of a run and hands out its bits; whenever 32 q have gathered they take the
// base-2 test, and whenever 32 have passed it, the Lucas test; the bits of
// those that fail are cleared.  Both lists carry over from run to run, so the
// tests run with all lanes at work.  A word is read, and its bits cleared, by
// one warp only.  Bound: the multiplier (prp64.cuh).
constexpr int kWinTestThreads = 256;
struct WinTestWarp {
  uint64_t cq[64], cat[64];  // to test: q and its bit in the masks
  uint64_t pq[64], pat[64];  // passed base 2
};

__global__ void __launch_bounds__(kWinTestThreads, kWinTestCtasPerSm)
    win_test_kernel(const __grid_constant__ WinTestArgs a) {
  constexpr uint32_t kAll = 0xffffffffu;
  __shared__ WinTestWarp s_warp[kWinTestThreads / 32];
  WinTestWarp& s = s_warp[threadIdx.x >> 5];
  const int lane = threadIdx.x & 31;
  const uint32_t below = (1u << lane) - 1;
  // runs per fetch: enough to spread the runs over the warps eight times
  const uint64_t warps = (uint64_t)gridDim.x * (kWinTestThreads / 32);
  const uint64_t step = a.runs / (8 * warps) + 1;
  uint64_t run = 0, run_end = 0;
  uint32_t w = 0, word = 0, nc = 0, np = 0;
  uint64_t q0 = 0, at0 = 0;  // the q and the place of the word's bit 0
  bool done = false;
  for (;;) {
    while (nc < 32 && !done) {
      if (!__any_sync(kAll, word != 0)) {  // the next run
        if (run == run_end) {
          unsigned long long r = 0;
          if (lane == 0) r = atomicAdd(a.ctr, (unsigned long long)step);
          run = __shfl_sync(kAll, r, 0);
          if (run >= a.runs) {
            done = true;
            break;
          }
          run_end = run + step < a.runs ? run + step : a.runs;
          w = find_item_window(a.run_off, a.nwin, run);
        }
        while (a.run_off[w + 1] <= run) ++w;
        const WinDesc6& d = a.win[w];
        const uint32_t lwords = d.lwords, runs = (lwords + 31) / 32;
        const uint32_t r = (uint32_t)(run - a.run_off[w]);
        const uint32_t c5 = r >= runs;
        const uint32_t t = 32 * (c5 ? r - runs : r) + lane;
        const uint64_t at = d.lbase + (c5 ? lwords : 0) + t;
        word = t < lwords ? a.lmask[at] : 0;
        q0 = 6 * ((uint64_t)d.g0 + 32ull * t) + (c5 ? 5 : 1);
        at0 = 32 * at;
        ++run;
        continue;
      }
      const uint32_t b = __ballot_sync(kAll, word != 0);
      if (word) {
        const int j = __ffs(word) - 1;
        word &= word - 1;
        const uint32_t i = nc + __popc(b & below);
        s.cq[i] = q0 + 6 * j;
        s.cat[i] = at0 + j;
      }
      nc += __popc(b);
    }
    if (nc) {
      const uint32_t m = min(nc, 32u);
      nc -= m;
      __syncwarp();
      const bool act = lane < (int)m;
      const uint64_t q = act ? s.cq[nc + lane] : 3, at = act ? s.cat[nc + lane] : 0;
      const bool pass = sprp2_any(q, act) && act;
      const uint32_t b = __ballot_sync(kAll, pass);
      if (pass) {
        const uint32_t i = np + __popc(b & below);
        s.pq[i] = q;
        s.pat[i] = at;
      } else if (act) {
        atomicAnd(&a.lmask[at >> 5], ~(1u << (at & 31)));
      }
      np += __popc(b);
      __syncwarp();
    }
    if (np >= 32 || (done && nc == 0 && np)) {
      const uint32_t m = min(np, 32u);
      np -= m;
      const bool act = lane < (int)m;
      const uint64_t q = act ? s.pq[np + lane] : 3, at = act ? s.pat[np + lane] : 0;
      if (!lucas_any(q, act) && act) atomicAnd(&a.lmask[at >> 5], ~(1u << (at & 31)));
      __syncwarp();
    }
    if (done && nc == 0 && np == 0) break;
  }
}

cudaError_t launch_win_test(const WinTestArgs& a, int grid, cudaStream_t s) {
  win_test_kernel<<<grid, kWinTestThreads, 0, s>>>(a);
  return cudaGetLastError();
}

// Windows that go n by n: the n of each window, laid out
// window after window at off[i], for the single-n kernel.
__global__ void win_expand_kernel(const gb_window* __restrict__ w, const uint64_t* __restrict__ off,
                                  uint32_t nw, uint64_t* __restrict__ n) {
  for (uint32_t i = blockIdx.x; i < nw; i += gridDim.x) {
    const uint64_t s = w[i].start, c = w[i].count, o = off[i];
    for (uint64_t j = threadIdx.x; j < c; j += blockDim.x) n[o + j] = s + 2 * j;
  }
}

cudaError_t launch_win_expand(const gb_window* w, const uint64_t* off, uint32_t nw, uint64_t* n,
                              cudaStream_t s) {
  if (!nw) return cudaSuccess;
  win_expand_kernel<<<nw < 4096 ? nw : 4096, 256, 0, s>>>(w, off, nw, n);
  return cudaGetLastError();
}

}  // namespace gb
