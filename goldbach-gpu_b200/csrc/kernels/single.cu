// single.cu -- batched single-n minimal partitions and batched primality.
//
// Replaces goldbach_single_kernel + check_single (src/single_check.cu:
// 95-282).  The reference sieves p in chunks of 1e8 on the CPU, copies them
// to the GPU, runs one thread per p with a 128-bit-remainder Miller-Rabin
// and keeps whichever thread finishes first, so its p is not the minimal
// one.  Here a query n walks the candidate primes p = 3, 5, 7, ... in order
// until q = n - p is prime:
//   1. the first 64 candidates (p <= 313) are sieved at once: for each odd
//      prime r <= 617, the residue of n mod r picks a 64-bit mask of the
//      candidates whose q r does not divide (SieveTab), and the masks are
//      ANDed; about 3.8 survivors are then tested per query near 2^63;
//   2. a survivor's q takes the base-2 strong test, 32 lanes at once with the
//      loops uniform across the warp (prp64.cuh);
//   3. a pass takes the extra strong Lucas test, which makes it a proof.
// A warp holds up to 32 queries and deals its lanes out to them: with 32
// queries each has one lane (throughput), with fewer each has several, which
// test that many of its survivors at once (latency, and the tail of a large
// batch).  Queries n < 2^21 (where q may be a prime <= 617) take a
// warp-cooperative scan with the full test per candidate.
#include <cuda_runtime.h>

#include <cstdint>
#include <type_traits>

#include "../gb_device.cuh"
#include "../gb_internal.h"
#include "prp64.cuh"

namespace gb {

constexpr uint64_t kSmallN = 1ull << 21;  // below this, q may be tiny: plain path
constexpr uint32_t kFull = 0xffffffffu;

__device__ __forceinline__ uint32_t lanemask_lt() {
  uint32_t m;
  asm("mov.u32 %0, %%lanemask_lt;" : "=r"(m));
  return m;
}

// Lane-parallel ascending scan over the primes above p_after with the full
// primality test per lane (the whole warp serves one n).
__device__ __noinline__ uint32_t minp_plain(const SingleArgs& a, uint64_t n, uint32_t p_after) {
  const int lane = threadIdx.x & 31;
  const uint64_t half = n >> 1;
  const uint64_t lim = half < a.p_lim ? half : a.p_lim;
  for (uint64_t k = 1;; k += 32) {
    const uint64_t kk = k + lane;
    const uint32_t p = kk < a.nprimes ? a.primes[kk] : 0xffffffffu;
    const bool valid = kk < a.nprimes && p <= lim;
    const bool ok = valid && p > p_after && is_prime_u64(n - p);
    const uint32_t b = __ballot_sync(kFull, ok);
    if (b) return __shfl_sync(kFull, p, __ffs(b) - 1);
    if (__ballot_sync(kFull, valid) != kFull) return 0;
  }
}

// Exact division by an odd r on 32-bit x: x * r^-1 (mod 2^32) lands in
// [0, (2^32-1)/r] exactly for the multiples of r.
__host__ __device__ constexpr uint32_t inv32(uint32_t r) {
  uint32_t x = r;  // r*r == 1 (mod 8)
  for (int i = 0; i < 4; ++i) x *= 2u - r * x;
  return x;
}
template <uint32_t R>
__device__ __forceinline__ bool divides(uint32_t x) {
  constexpr uint32_t kInv = inv32(R), kLim = 0xffffffffu / R;
  static_assert(R * kInv == 1u, "inverse");
  return x * kInv <= kLim;
}

constexpr uint32_t kM1 = 3u * 5 * 7 * 11 * 13 * 17 * 19 * 23;  // 111546435
constexpr uint32_t kM2 = 29u * 31 * 37 * 41 * 43;              // 58642669
constexpr uint32_t kM3 = 47u * 53 * 59 * 61;                   // 8965109

// q = n - p has no prime factor <= 61, from n mod M1, M2, M3.
__device__ __forceinline__ bool no_small_factor(uint32_t nm1, uint32_t nm2, uint32_t nm3,
                                                uint32_t p) {
  uint32_t x = nm1 + kM1 - p % kM1;
  x = x >= kM1 ? x - kM1 : x;
  bool f = divides<3>(x) | divides<5>(x) | divides<7>(x) | divides<11>(x) | divides<13>(x) |
           divides<17>(x) | divides<19>(x) | divides<23>(x);
  uint32_t y = nm2 + kM2 - p % kM2;
  y = y >= kM2 ? y - kM2 : y;
  f |= divides<29>(y) | divides<31>(y) | divides<37>(y) | divides<41>(y) | divides<43>(y);
  uint32_t z = nm3 + kM3 - p % kM3;
  z = z >= kM3 ? z - kM3 : z;
  f |= divides<47>(z) | divides<53>(z) | divides<59>(z) | divides<61>(z);
  return !f;
}

// The candidate sieve.  Bit k of a mask stands for the k-th odd prime p (3, 5,
// ..., 313).  For each of the first kSieveMods moduli R -- a prime up to 313, or a
// product of a few small ones -- a table gives the mask of x = n mod R: bit k
// is clear when a prime factor f of R divides x - p, that is when f divides
// q = n - p.  A prime r above 313 strikes at most the candidate p = n mod r
// itself, so those up to 617 share one table of 315 masks (kSieveOnes; the
// last entry strikes nothing).  617 is about where one more prime (15 clocks
// a lane) stops paying for the base-2 tests it saves (4 x 3900 / r clocks).
constexpr int kSieveMods = 57;
__host__ __device__ constexpr uint32_t sieve_mod(int i) {
  constexpr uint16_t kMods[kSieveMods] = {
      1155, 221, 437, 899, 1517, 43,  47,  53,  59,  61,  67,  71,  73,  79,  83,  89,  97,  101, 103,
      107,  109, 113, 127, 131,  137, 139, 149, 151, 157, 163, 167, 173, 179, 181, 191, 193, 197, 199,
      211,  223, 227, 229, 233,  239, 241, 251, 257, 263, 269, 271, 277, 281, 283, 293, 307, 311, 313};
  return kMods[i];
}
__host__ __device__ constexpr uint32_t sieve_offset(int i) {
  uint32_t o = 0;
  for (int j = 0; j < i; ++j) o += sieve_mod(j);
  return o;
}
constexpr uint32_t kSieveOnes = sieve_offset(kSieveMods);
constexpr uint32_t kSieveEntries = kSieveOnes + 315;

struct SieveTab {
  uint64_t m[kSieveEntries];
  uint64_t m2[kSieveOnes];  // the same for the next 64 odd primes (317, ..., 727)
  uint32_t mod[kSieveMods], off[kSieveMods];
  constexpr SieveTab() : m(), m2(), mod(), off() {
    uint32_t odd_primes[128] = {};
    int np = 0;
    for (uint32_t v = 3; np < 128; v += 2) {
      bool prime = true;
      for (int k = 0; k < np && prime; ++k) prime = v % odd_primes[k] != 0;
      if (prime) odd_primes[np++] = v;
    }
    for (uint32_t i = 0; i < kSieveEntries; ++i) m[i] = ~0ull;
    for (uint32_t i = 0; i < kSieveOnes; ++i) m2[i] = ~0ull;
    uint32_t o = 0;
    for (int i = 0; i < kSieveMods; ++i) {
      const uint32_t R = sieve_mod(i);
      mod[i] = R;
      off[i] = o;
      for (int j = 0; j < 64; ++j) {  // prime factors of R (all <= 313)
        const uint32_t f = odd_primes[j];
        if (R % f) continue;
        for (int k = 0; k < 64; ++k)
          for (uint32_t x = odd_primes[k] % f; x < R; x += f) m[o + x] &= ~(1ull << k);
        for (int k = 0; k < 64; ++k)
          for (uint32_t x = odd_primes[64 + k] % f; x < R; x += f) m2[o + x] &= ~(1ull << k);
      }
      o += R;
    }
    for (int k = 0; k < 64; ++k) m[kSieveOnes + odd_primes[k]] &= ~(1ull << k);
  }
};
__device__ const SieveTab g_sieve{};

// n mod M for a constant 2^16 < M < 2^31 from one FMA of n as a double: the
// conversion and 1/M are each within 2^-53 of exact, so before the sum is rounded
// the estimate is within 2^-4 of n / M < 2^48 and rounds to floor(n / M) or one
// more; the low 32 bits of the sum with 1.5 * 2^52 are that quotient's.
template <uint32_t M>
__device__ __forceinline__ uint32_t mod_const(double nd, uint32_t nl) {
  static_assert(M > (1u << 16) && M < (1u << 31), "quotient estimate");
  constexpr double kInv = 1.0 / M;
  const uint32_t qt = (uint32_t)__double_as_longlong(fma(nd, kInv, 6755399441055744.0));
  const uint32_t r = nl - qt * M;
  return min(r, r + M);
}

// The masks of C moduli from index I on, by way of n mod their product.
template <int I, int C>
__device__ __forceinline__ uint64_t sieve_group(const uint64_t* tab, double nd, uint32_t nl) {
  constexpr uint32_t M = sieve_mod(I) * (C > 1 ? sieve_mod(I + (C > 1)) : 1u) *
                         (C > 2 ? sieve_mod(I + 2 * (C > 2)) : 1u) *
                         (C > 3 ? sieve_mod(I + 3 * (C > 3)) : 1u);
  const uint32_t x = mod_const<M>(nd, nl);
  uint64_t m = tab[sieve_offset(I) + x % sieve_mod(I)];
  if constexpr (C > 1) m &= tab[sieve_offset(I + 1) + x % sieve_mod(I + 1)];
  if constexpr (C > 2) m &= tab[sieve_offset(I + 2) + x % sieve_mod(I + 2)];
  if constexpr (C > 3) m &= tab[sieve_offset(I + 3) + x % sieve_mod(I + 3)];
  return m;
}
// The same for three primes above 313.
template <uint32_t A, uint32_t B, uint32_t C>
__device__ __forceinline__ uint64_t sieve_ones(const uint64_t* tab, double nd, uint32_t nl) {
  const uint32_t x = mod_const<A * B * C>(nd, nl);
  const uint64_t* t = tab + kSieveOnes;
  return t[min(x % A, 314u)] & t[min(x % B, 314u)] & t[min(x % C, 314u)];
}

__device__ __forceinline__ uint64_t sieve_all(const uint64_t* tab, uint64_t n) {
  const double nd = __ull2double_rn(n);
  const uint32_t nl = (uint32_t)n;
  uint64_t m = sieve_group<0, 3>(tab, nd, nl) & sieve_group<3, 3>(tab, nd, nl) &
               sieve_group<6, 4>(tab, nd, nl) & sieve_group<10, 4>(tab, nd, nl) &
               sieve_group<14, 4>(tab, nd, nl) & sieve_group<18, 4>(tab, nd, nl) &
               sieve_group<22, 4>(tab, nd, nl) & sieve_group<26, 4>(tab, nd, nl) &
               sieve_group<30, 4>(tab, nd, nl) & sieve_group<34, 4>(tab, nd, nl) &
               sieve_group<38, 3>(tab, nd, nl) & sieve_group<41, 3>(tab, nd, nl) &
               sieve_group<44, 3>(tab, nd, nl) & sieve_group<47, 3>(tab, nd, nl) &
               sieve_group<50, 3>(tab, nd, nl) & sieve_group<53, 2>(tab, nd, nl) &
               sieve_group<55, 2>(tab, nd, nl);
  m &= sieve_ones<317, 331, 337>(tab, nd, nl) & sieve_ones<347, 349, 353>(tab, nd, nl) &
       sieve_ones<359, 367, 373>(tab, nd, nl) & sieve_ones<379, 383, 389>(tab, nd, nl) &
       sieve_ones<397, 401, 409>(tab, nd, nl) & sieve_ones<419, 421, 431>(tab, nd, nl) &
       sieve_ones<433, 439, 443>(tab, nd, nl) & sieve_ones<449, 457, 461>(tab, nd, nl) &
       sieve_ones<463, 467, 479>(tab, nd, nl) & sieve_ones<487, 491, 499>(tab, nd, nl) &
       sieve_ones<503, 509, 521>(tab, nd, nl) & sieve_ones<523, 541, 547>(tab, nd, nl) &
       sieve_ones<557, 563, 569>(tab, nd, nl) & sieve_ones<571, 577, 587>(tab, nd, nl) &
       sieve_ones<593, 599, 601>(tab, nd, nl) & sieve_ones<607, 613, 617>(tab, nd, nl);
  return m;
}

// The warp's sieve of the first 128 candidates of one n (lanes agree on n)
// over the moduli with tables of their own, for small batches: a query's
// lanes test more survivors at once than 64 candidates leave (about 17), and
// the few queries whose minimal p lies beyond 313 (6%) would make the whole
// batch wait for further rounds (100 queries: 41 -> 28 us).
struct Mask128 {
  uint64_t lo, hi;
};
__device__ __forceinline__ uint64_t warp_and(uint64_t m) {
  const uint32_t l = __reduce_and_sync(kFull, (uint32_t)m), h = __reduce_and_sync(kFull, (uint32_t)(m >> 32));
  return (uint64_t)h << 32 | l;
}
__device__ __forceinline__ Mask128 sieve_warp(uint64_t n) {
  const uint32_t hi = (uint32_t)(n >> 32), lo = (uint32_t)n;
  Mask128 m{~0ull, ~0ull};
#pragma unroll 1
  for (int j = threadIdx.x & 31; j < kSieveMods; j += 32) {
    const uint32_t R = g_sieve.mod[j];
    // n mod R from its halves: R < 2^11, so the sum stays below 2^32
    const uint32_t t = g_sieve.off[j] + ((hi % R) * ((0xffffffffu % R + 1) % R) + lo % R) % R;
    m.lo &= g_sieve.m[t];
    m.hi &= g_sieve.m2[t];
  }
  return {warp_and(m.lo), warp_and(m.hi)};
}

// Bits of the 64 candidates from prime index k0 on that are <= p_lim: a whole
// warp's call, two loads a lane.
__device__ __forceinline__ uint64_t candidates_below(const SingleArgs& a, uint32_t k0) {
  const uint32_t k = k0 + (threadIdx.x & 31);
  const uint32_t lo = __ballot_sync(kFull, k < a.nprimes && a.primes[k] <= a.p_lim);
  const uint32_t hi = __ballot_sync(kFull, k + 32 < a.nprimes && a.primes[k + 32] <= a.p_lim);
  return (uint64_t)hi << 32 | lo;
}

// Every round the warp deals its 32 lanes out to its A <= 32 queries (slots),
// rank by rank: lane l tests survivor l / A of query l % A.  The lowest rank
// that passes base 2 holds the query's minimal candidate; it joins the warp's
// pending list and the slot is free for the next query at once.  Whenever 32
// candidates are pending, one Lucas test proves them all, so both tests run
// with (nearly) all lanes at work, and the sieve runs for a whole warp's
// refill of queries at a time.  A candidate that the Lucas test rejects (a
// base-2 pseudoprime) sends its query through minp_plain from there on.
//
// Bound: the multiplier (prp64.cuh).  One CTA of 16 warps per SM: four warps
// per quarter cover a product's latency (95 clocks against 54 of issue), and
// the sieve tables take 108 KB. 
// Device time of a batch uniform below 2^64, against one strong test to each
// of 7 bases on a lane (8192 queries or more) or a warp (fewer) per query:
// 1e6 queries 2.97 -> 0.97 ms, 20000 648 -> 81 us, 8191 107 -> 57, 3001 58 -> 47,
// 592 and fewer unchanged (36 us, of which about 13 are the launch).
constexpr int kSingleThreads = 512;
struct SingleWarp {
  // slots: query, its index, its survivors not yet tested among 128 candidates,
  // prime index of mask's bit 0, and of the next block (0: none)
  uint64_t n[32], qi[32], mask[32], mask2[32];
  uint32_t cbase[32], kb[32];
  uint64_t rn[32], rmask[32], rmask2[32], rqi[32];  // sieved queries not yet in a slot
  uint64_t pq[64], pqi[64];          // pending: q, query index
  uint32_t pp[64];                   // and p
  uint32_t slot[32];                 // the occupied slots in order
};
constexpr int kSingleWarps = kSingleThreads / 32;
struct SingleCta {
  SingleWarp warp[kSingleWarps];
  uint64_t pq[31 * kSingleWarps], pqi[31 * kSingleWarps];  // pending at the end
  uint32_t pp[31 * kSingleWarps], npend;
};
constexpr size_t kSingleTabBytes = kSieveEntries * sizeof(uint64_t);

// Clears the lowest set bit of hi : lo.
__device__ __forceinline__ void drop_lowest(uint64_t& lo, uint64_t& hi) {
  if (lo) lo &= lo - 1;
  else hi &= hi - 1;
}

template <bool STAGED>
__global__ void __launch_bounds__(kSingleThreads, 1) single_kernel(SingleArgs a) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  SingleCta& cta = *reinterpret_cast<SingleCta*>(smem_raw);
  SingleWarp& w = cta.warp[threadIdx.x >> 5];
  uint64_t* tab = reinterpret_cast<uint64_t*>(smem_raw + sizeof(SingleCta));
  if (STAGED)
    for (uint32_t i = threadIdx.x; i < kSieveEntries; i += kSingleThreads) tab[i] = g_sieve.m[i];
  if (threadIdx.x == 0) cta.npend = 0;
  __syncthreads();
  const int lane = threadIdx.x & 31;
  const uint64_t mask0 = candidates_below(a, 1), mask1 = STAGED ? 0 : candidates_below(a, 65);
  // the block after a slot's masks, 0 when p_lim ends among them
  const uint32_t kb0 = STAGED ? (mask0 == ~0ull ? 65 : 0) : (mask1 == ~0ull ? 129 : 0);
  const uint32_t chunk = a.warp_queries;  // queries a warp holds, 1 .. 32
  uint32_t active = 0, nready = 0, npend = 0;
  bool first = true, drained = false;
  uint32_t found = 0, maxp = 0;
  auto finish = [&](uint64_t i, uint32_t pf, uint64_t q) {
    a.p_out[i] = pf;
    a.q_out[i] = q;
    if (pf) {
      ++found;
      maxp = pf > maxp ? pf : maxp;
    }
  };
  // Lucas tests of the lanes' q = n - p (PAIR: lanes 2i and 2i + 1 hold the same)
  auto prove = [&](uint64_t q, uint64_t i, uint32_t p, bool act, auto pair) {
    constexpr bool PAIR = decltype(pair)::value;
    const bool ok = PAIR ? lucas_pair_any(q, act) : lucas_any(q, act);
    if (PAIR && (lane & 1)) act = false;
    if (act && ok) finish(i, p, q);
    for (uint32_t bad = __ballot_sync(kFull, act && !ok); bad; bad &= bad - 1) {
      const int l = __ffs(bad) - 1;
      const uint64_t n = __shfl_sync(kFull, q + p, l);
      const uint32_t pl = minp_plain(a, n, __shfl_sync(kFull, p, l));
      if (lane == l) finish(i, pl, pl ? n - pl : 0);
    }
    __syncwarp();
  };
  for (;;) {
    // fill the slots
    for (;;) {
      if (nready == 0 && !drained && (uint32_t)__popc(active) < chunk) {
        // the first queries by place, the others from the work counter
        const uint64_t warps = (uint64_t)gridDim.x * kSingleWarps;
        unsigned long long base = 0;
        if (first) {
          base = ((uint64_t)(threadIdx.x >> 5) * gridDim.x + blockIdx.x) * chunk;
        } else {
          if (lane == 0) base = warps * chunk + atomicAdd(&a.ctr[0], (unsigned long long)chunk);
          base = __shfl_sync(kFull, base, 0);
        }
        first = false;
        drained = base >= a.count;
        const uint64_t qi = base + lane;
        bool ready = lane < (int)chunk && qi < a.count;
        const uint64_t n = ready ? a.n[qi] : 0;
        if (ready && (n <= 4 || (n & 1))) {
          finish(qi, n == 4 ? 2 : 0, n == 4 ? 2 : 0);
          ready = false;
        }
        const uint32_t rb = __ballot_sync(kFull, ready);
        uint64_t m = 0, m2 = 0;
        if (STAGED) {
          if (ready && n >= kSmallN) m = sieve_all(tab, n) & mask0;
        } else {
          for (uint32_t left = __ballot_sync(kFull, ready && n >= kSmallN); left; left &= left - 1) {
            const int l = __ffs(left) - 1;
            const Mask128 ml = sieve_warp(__shfl_sync(kFull, n, l));
            if (lane == l) {
              m = ml.lo & mask0;
              m2 = ml.hi & mask1;
            }
          }
        }
        if (ready) {
          const uint32_t i = __popc(rb & lanemask_lt());
          w.rn[i] = n;
          w.rmask[i] = m;
          if (!STAGED) w.rmask2[i] = m2;
          w.rqi[i] = qi;
        }
        nready = __popc(rb);
        __syncwarp();
      }
      // ready queries into free slots (slots 0 .. chunk - 1 are in use)
      const uint32_t room = ~active & (chunk == 32 ? kFull : (1u << chunk) - 1);
      const uint32_t k = min((uint32_t)__popc(room), nready);
      const uint32_t rank = __popc(room & lanemask_lt());
      const bool take = ((room >> lane) & 1u) && rank < k;
      if (take) {
        const uint32_t i = nready - 1 - rank;
        w.n[lane] = w.rn[i];
        w.mask[lane] = w.rmask[i];
        if (!STAGED) w.mask2[lane] = w.rmask2[i];
        w.qi[lane] = w.rqi[i];
        w.cbase[lane] = 1;
        w.kb[lane] = kb0;
      }
      nready -= k;
      active |= __ballot_sync(kFull, take);
      __syncwarp();
      // slots without a survivor: further blocks of candidates, and small n
      for (;;) {
        const uint32_t b = __ballot_sync(kFull, ((active >> lane) & 1u) && (STAGED ? w.mask[lane] : w.mask[lane] | w.mask2[lane]) == 0);
        if (!b) break;
        const int j = __ffs(b) - 1;
        const uint64_t n = w.n[j];
        const uint32_t kj = w.kb[j];
        __syncwarp();
        if (n < kSmallN || kj == 0) {
          const uint32_t p = n < kSmallN ? minp_plain(a, n, 2) : 0;
          if (lane == j) finish(w.qi[j], p, p ? n - p : 0);  // kj = 0: every prime p <= p_lim tried
          active &= ~(1u << j);
          continue;
        }
        const uint64_t half = n >> 1;
        const uint32_t lim = (uint32_t)(half < a.p_lim ? half : a.p_lim);
        // a block is 64 candidates, or 128 when few queries wait for each other
        uint64_t blk[2] = {0, 0};
        uint32_t more = kFull;
#pragma unroll 1
        for (int i = 0; i < (STAGED ? 2 : 4) && more == kFull; ++i) {
          const uint64_t k = (uint64_t)kj + 32 * i + lane;
          const uint32_t pk = k < a.nprimes ? a.primes[k] : 0xffffffffu;
          const bool valid = k < a.nprimes && pk <= lim;
          const uint64_t pass = __ballot_sync(kFull, valid && no_small_factor(n % kM1, n % kM2, n % kM3, pk));
          more = __ballot_sync(kFull, valid);
          if (i < 2) blk[0] |= pass << (32 * i);
          else blk[1] |= pass << (32 * (i - 2));
        }
        if (lane == j) {
          w.mask[j] = blk[0];
          if (!STAGED) w.mask2[j] = blk[1];
          w.cbase[j] = kj;
          w.kb[j] = more == kFull ? kj + (STAGED ? 64 : 128) : 0;
        }
        __syncwarp();
      }
      if ((uint32_t)__popc(active) == chunk || (drained && nready == 0)) break;
    }
    if (active) {
      // deal the lanes out
      const uint32_t A = __popc(active);
      if ((active >> lane) & 1u) w.slot[__popc(active & lanemask_lt())] = lane;
      __syncwarp();
      const uint32_t idx = lane % A, rank = lane / A;
      const uint32_t j = w.slot[idx];
      uint64_t m = w.mask[j], m2 = STAGED ? 0 : w.mask2[j];
      for (uint32_t i = 0; i < 31 / A; ++i)
        if (i < rank) drop_lowest(m, m2);
      const bool act = (m | m2) != 0;
      const uint32_t bit = m ? __ffsll((long long)m) - 1 : 63 + __ffsll((long long)m2);
      const uint32_t p = act ? a.primes[w.cbase[j] + bit] : 0;
      const uint64_t q = act ? w.n[j] - p : 3;
      const bool pass = sprp2_any(q, act) && act;
      const uint32_t b = __ballot_sync(kFull, pass);
      uint32_t mine = 0;  // the lanes of this lane's query
      for (uint32_t i = idx; i < 32; i += A) mine |= 1u << i;
      const uint32_t win = b & mine;
      const int l = win ? __ffs(win) - 1 : lane;
      const uint64_t qw = __shfl_sync(kFull, q, l);
      const uint32_t pw = __shfl_sync(kFull, p, l);
      const uint32_t wb = __ballot_sync(kFull, rank == 0 && win);
      __syncwarp();
      if (rank == 0) {
        if (win) {
          const uint32_t i = npend + __popc(wb & lanemask_lt());
          w.pq[i] = qw;
          w.pqi[i] = w.qi[j];
          w.pp[i] = pw;
        } else {
          uint64_t left = w.mask[j], left2 = STAGED ? 0 : w.mask2[j];
          for (int i = __popc(mine); i > 0; --i) drop_lowest(left, left2);
          w.mask[j] = left;
          if (!STAGED) w.mask2[j] = left2;
        }
      }
      active &= ~__reduce_or_sync(kFull, rank == 0 && win ? 1u << j : 0u);
      npend += __popc(wb);
      // the rank-0 lanes' entries and masks before other lanes read them: the proof
      // below, the refill above, and the copy of what is left after the loop
      __syncwarp();
    }
    if (npend >= 32) {
      npend -= 32;
      prove(w.pq[npend + lane], w.pqi[npend + lane], w.pp[npend + lane], true, std::false_type{});
    }
    if (!active && drained && nready == 0) break;
  }
  // what the warps still have pending, proved 16 to a warp with a pair of lanes each
  uint32_t base = 0;
  if (lane == 0 && npend) base = atomicAdd(&cta.npend, npend);
  base = __shfl_sync(kFull, base, 0);
  if (lane < (int)npend) {
    cta.pq[base + lane] = w.pq[lane];
    cta.pqi[base + lane] = w.pqi[lane];
    cta.pp[base + lane] = w.pp[lane];
  }
  __syncthreads();
  const uint32_t total = cta.npend;
  for (uint32_t e0 = 16 * (threadIdx.x >> 5); e0 < total; e0 += 16 * kSingleWarps) {
    const uint32_t e = e0 + (lane >> 1);
    const bool act = e < total;
    prove(act ? cta.pq[e] : 3, act ? cta.pqi[e] : 0, act ? cta.pp[e] : 0, act, std::true_type{});
  }
  // the warp's counts, one atomic each
  found = __reduce_add_sync(kFull, found);
  maxp = __reduce_max_sync(kFull, maxp);
  if (lane == 0) {
    if (found) atomicAdd(&a.ctr[1], (unsigned long long)found);
    if (maxp) atomicMax(&a.ctr[2], (unsigned long long)maxp);
  }
}

// Shape of a batch on sm_count SMs, of which it may fill share_pct percent: the
// queries spread over 16 warps per SM, up to 32 each.  From kSingleTabQueries a
// warp on, the sieve tables are staged in shared memory and every lane sieves
// its own query: 20000 queries (9 a warp) take 81 us unstaged and 97 staged, 76000
// (32 a warp) 146 both ways, 40000 (17 a warp) 118 unstaged.
constexpr uint64_t kSpreadWarps = 16, kSingleTabQueries = 20;

struct SingleShape {
  void (*kernel)(SingleArgs);
  int grid;
  size_t smem;
};
static SingleShape single_shape(SingleArgs& a, int sm_count, uint32_t share_pct) {
  uint64_t sms = (uint64_t)sm_count * share_pct / 100;
  if (sms < 1) sms = 1;
  const uint64_t per = (a.count + sms * kSpreadWarps - 1) / (sms * kSpreadWarps);
  a.warp_queries = per < 1 ? 1 : per > 32 ? 32 : (uint32_t)per;
  const uint64_t need = (a.count + a.warp_queries - 1) / a.warp_queries;  // warps with a query
  const bool staged = per >= kSingleTabQueries;
  SingleShape s;
  s.kernel = staged ? single_kernel<true> : single_kernel<false>;
  s.grid = (int)(need < sms ? (need ? need : 1) : sms);
  s.smem = sizeof(SingleCta) + (staged ? kSingleTabBytes : 0);
  cudaFuncSetAttribute(s.kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)s.smem);
  return s;
}

cudaError_t launch_single(const SingleArgs& args, int sm_count, uint32_t share_pct, cudaStream_t s) {
  SingleArgs a = args;
  const SingleShape sh = single_shape(a, sm_count, share_pct);
  sh.kernel<<<sh.grid, kSingleThreads, sh.smem, s>>>(a);
  return cudaGetLastError();
}

void single_kernel_node(SingleArgs& a, int sm_count, void** argv, cudaKernelNodeParams* kp) {
  const SingleShape sh = single_shape(a, sm_count, 100);
  argv[0] = (void*)&a;
  *kp = cudaKernelNodeParams{};
  kp->func = (void*)sh.kernel;
  kp->gridDim = dim3((unsigned)sh.grid);
  kp->blockDim = dim3(kSingleThreads);
  kp->sharedMemBytes = (unsigned)sh.smem;
  kp->kernelParams = argv;
}

// Per-request totals of a single-lane batch: request r owns the n of
// [off[r], off[r+1]); agg[4r..4r+3] = verified, failures, max p, sum of p.
__global__ void segment_reduce_kernel(const uint64_t* p, const uint64_t* off, uint32_t nreq,
                                      unsigned long long* agg) {
  const uint32_t r = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int lane = threadIdx.x & 31;
  if (r >= nreq) return;
  unsigned long long v = 0, f = 0, mx = 0, sum = 0;
  for (uint64_t i = off[r] + lane; i < off[r + 1]; i += 32) {
    const uint64_t x = p[i];
    if (x) {
      ++v;
      sum += x;
      if (x > mx) mx = x;
    } else {
      ++f;
    }
  }
  for (int o = 16; o; o >>= 1) {
    v += __shfl_down_sync(0xffffffffu, v, o);
    f += __shfl_down_sync(0xffffffffu, f, o);
    sum += __shfl_down_sync(0xffffffffu, sum, o);
    const unsigned long long m2 = __shfl_down_sync(0xffffffffu, mx, o);
    if (m2 > mx) mx = m2;
  }
  if (lane == 0) {
    agg[4 * r] = v;
    agg[4 * r + 1] = f;
    agg[4 * r + 2] = mx;
    agg[4 * r + 3] = sum;
  }
}

cudaError_t launch_segment_reduce(const uint64_t* p, const uint64_t* off, uint32_t nreq,
                                  unsigned long long* agg, cudaStream_t s) {
  if (!nreq) return cudaSuccess;
  segment_reduce_kernel<<<(nreq + 7) / 8, 256, 0, s>>>(p, off, nreq, agg);
  return cudaGetLastError();
}

void segment_reduce_node(const SegReduceArgs& r, void** argv, cudaKernelNodeParams* kp) {
  argv[0] = (void*)&r.p;
  argv[1] = (void*)&r.off;
  argv[2] = (void*)&r.nreq;
  argv[3] = (void*)&r.agg;
  *kp = cudaKernelNodeParams{};
  kp->func = (void*)segment_reduce_kernel;
  kp->gridDim = dim3((r.nreq + 7) / 8);
  kp->blockDim = dim3(256);
  kp->kernelParams = argv;
}

__global__ void is_prime_kernel(const uint64_t* n, uint64_t count, uint8_t* out) {
  for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < count;
       i += (uint64_t)gridDim.x * blockDim.x)
    out[i] = is_prime_u64(n[i]) ? 1 : 0;
}

cudaError_t launch_is_prime(const uint64_t* n, uint64_t count, uint8_t* out, cudaStream_t s) {
  if (!count) return cudaSuccess;
  uint64_t blocks = (count + 255) / 256;
  if (blocks > 148 * 32) blocks = 148 * 32;
  is_prime_kernel<<<(unsigned)blocks, 256, 0, s>>>(n, count, out);
  return cudaGetLastError();
}

}  // namespace gb
