// big.cu -- Goldbach partitions of even n beyond 2^64 (multi-precision).
//
// Replaces big_check (src/big_check.cpp:35-144), which scans the primes up
// to 1e7 in OpenMP batches of 1000 and keeps the first q = n - p that GMP's
// mpz_probab_prime_p(q, 25) accepts -- a valid partition, not guaranteed
// the minimal one.  Here the candidates p (ascending, from the resident
// prime table) are tested in batches (host/gb_big.cpp):
//   1. big_filter_kernel: one warp per candidate drops q = n - p when a
//      trial prime r divides it, from n mod r (computed on the host once per
//      n) and p mod r; the survivors are a bitmap;
//   2. big_base2_kernel: one group of lanes per survivor runs the strong
//      probable-prime test to base 2, lists the passers (almost all of them
//      primes) and keeps the smallest; up to 1024 bits, more CTAs run the other
//      bases on the first survivors meanwhile;
//   3. big_bases_kernel: one warp per base runs the 11 other bases 3, 5, ...,
//      37 -- with base 2 the base set of the reference's Miller-Rabin
//      (src/goldbach.cu:333-360) -- on one passer.
// The smallest passer no base rejects is the minimal p: every smaller
// candidate was tested and failed.  The test is deterministic for
// q < 3.3e24 (the 12 prime bases admit no strong pseudoprime below that) and
// a probable-prime test beyond, like the reference's.
//
// A batch is a few hundred tests of hundreds to thousands of dependent
// products each, so the latency of one product is what bounds it, not the
// multiplier.  A number is therefore spread over G lanes, K limbs of 32 bits
// per lane (up to 32 limbs one a lane, G = 8, 16 or 32), and a product takes
// one step per limb of y: every lane multiplies its limbs by it, lane 0's
// lowest limb gives the reduction's m, and the limbs move down one place.
// A step is about 70 clocks (one round of shuffles, then two multiplications
// and the sums in a row), whatever the width.  The carries stay in 64-bit
// accumulators until the end, where one pass over the lanes and a carry
// look-ahead on two ballots settle them; R = 2^(32 L) >= 4q keeps the residues below 2q without a
// subtraction.  One n of 512 bits: 22.0 -> 0.6 ms (one thread per test with its
// limbs in local memory took 10.9 ms for each of the two strong-test kernels,
// 41,000 clocks a product; moving m, then the limbs, in two rounds of shuffles
// took 1.22 ms where this takes 1.03, both in batches of 8192 candidates).
#include <cuda_runtime.h>

#include <cstdint>
#include <type_traits>

#include "../gb_internal.h"

namespace gb {

constexpr uint32_t kAllLanes = 0xffffffffu;
constexpr int kBigMaxLimbs = GB_BIG_MAX_LIMBS + 1;  // limbs of R

// The 12 prime bases of the strong tests.
__device__ __constant__ const uint32_t kBigBases[12] = {2, 3, 5, 7, 11, 13, 17, 19, 23, 29, 31, 37};

// A warp per candidate, a word of a.surv per CTA.
constexpr int kFilterThreads = 1024;
__global__ void __launch_bounds__(kFilterThreads) big_filter_kernel(const __grid_constant__ BigArgs a, uint32_t k0,
                                                                    uint32_t kcount) {
  __shared__ uint32_t s_drop[32];
  const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t i = blockIdx.x * 32 + warp;
  bool drop = i >= kcount;  // warp-uniform
  if (!drop) {
    const uint32_t p = a.primes[k0 + i];
    drop = p > a.p_lim;
    for (uint32_t j = lane; j < a.ntrial; j += 32)
      drop |= p % a.trial[j] == a.nmod[j];  // r divides q = n - p (q far above r)
  }
  drop = __any_sync(kAllLanes, drop);
  if (lane == 0) s_drop[warp] = drop;
  __syncthreads();
  if (warp == 0) {
    const uint32_t w = __ballot_sync(kAllLanes, !s_drop[lane]);
    if (lane == 0) a.surv[blockIdx.x] = w;
  }
}

// The survivors by rank, from their bits: lane l holds the words [l per, (l + 1) per).
struct Survivors {
  const uint32_t* bits;
  uint32_t words, per, upto;  // upto: survivors up to this lane's words, included
  uint32_t total;

  __device__ __forceinline__ Survivors(const BigArgs& a)
      : bits(a.surv), words(a.words), per((a.words + 31) / 32), upto(0) {
    const uint32_t lane = threadIdx.x & 31;
    for (uint32_t j = lane * per; j < min((lane + 1) * per, words); ++j) upto += __popc(bits[j]);
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
      const uint32_t v = __shfl_up_sync(kAllLanes, upto, d);
      if (lane >= (uint32_t)d) upto += v;
    }
    total = __shfl_sync(kAllLanes, upto, 31);
  }
  // candidate index of survivor t (below total; t may differ between lanes)
  __device__ __forceinline__ uint32_t nth(uint32_t t) const {
    uint32_t own = 0, before = 0;  // the lane whose words hold it, the survivors below those
    for (int l = 0; l < 31; ++l) {
      const uint32_t v = __shfl_sync(kAllLanes, upto, l);
      if (t >= v) {
        own = l + 1;
        before = v;
      }
    }
    uint32_t j = own * per, w = bits[j];
    t -= before;
    for (uint32_t c; t >= (c = __popc(w)); w = bits[++j]) t -= c;
    for (; t; --t) w &= w - 1;
    return 32 * j + __ffs(w) - 1;
  }
  __device__ __forceinline__ uint32_t rank(uint32_t i) const {  // survivors below candidate i
    uint32_t c = 0;
    for (uint32_t j = threadIdx.x & 31; j <= i >> 5; j += 32)
      c += __popc(j < i >> 5 ? bits[j] : bits[j] & ((1u << (i & 31)) - 1));
    return __reduce_add_sync(kAllLanes, c);
  }
};

// candidate index of survivor t, or of the last one; ~0u without any (t may
// differ between lanes).  A call, so that a test's registers are its own (inlined:
// 4096 bits 104.5 -> 106.5 ms).
__device__ __noinline__ uint32_t nth_survivor(const BigArgs& a, uint32_t t) {
  const Survivors S(a);
  return S.total ? S.nth(min(t, S.total - 1)) : 0xffffffffu;
}

// Numbers of G lanes with K limbs each; limb j of lane l is limb l K + j.
template <int G, int K>
struct Big {
  typedef uint32_t Num[K];

  static __device__ __forceinline__ int sub() { return threadIdx.x & (G - 1); }
  static __device__ __forceinline__ uint32_t up(uint32_t v) {  // from the lane below (0 into lane 0)
    const uint32_t r = __shfl_up_sync(kAllLanes, v, 1, G);
    return sub() ? r : 0;
  }
  // The carry into this lane, from the lanes that generate one (g) and those
  // that pass one on (p, not g): the carries of the sum of two numbers whose
  // bits generate and propagate alike (carry look-ahead by one addition of the two
  // ballots, a known technique).  out: the carry out of the last lane.
  static __device__ __forceinline__ uint32_t carry_in(bool g, bool p, bool& out) {
    uint32_t gb = __ballot_sync(kAllLanes, g), pb = __ballot_sync(kAllLanes, p && !g);
    if (G < 32) {
      const int lead = (threadIdx.x & 31) & ~(G - 1);
      gb = (gb >> lead) & ((1u << (G & 31)) - 1);
      pb = (pb >> lead) & ((1u << (G & 31)) - 1);
    }
    const uint64_t s = (uint64_t)(gb | pb) + gb;
    out = (s >> G) & 1;
    return ((uint32_t)s ^ pb) >> sub() & 1;
  }
  // r = the number with the 64-bit limbs c (below R): c's high halves go to the
  // next limb.
  static __device__ __forceinline__ void settle(Num& r, uint64_t (&c)[K]) {
    uint64_t carry = 0;
#pragma unroll
    for (int j = 0; j < K; ++j) {
      c[j] += carry;  // (c stays far below 2^64: high halves of at most a few)
      r[j] = (uint32_t)c[j];
      carry = c[j] >> 32;
    }
    uint32_t in = up((uint32_t)carry);
    bool ones = true;
#pragma unroll
    for (int j = 0; j < K; ++j) {
      const uint64_t t = (uint64_t)r[j] + in;
      r[j] = (uint32_t)t;
      in = (uint32_t)(t >> 32);
      ones &= r[j] == 0xffffffffu;
    }
    bool out;
    in = carry_in(in != 0, ones, out);
#pragma unroll
    for (int j = 0; j < K; ++j) {
      const uint64_t t = (uint64_t)r[j] + in;
      r[j] = (uint32_t)t;
      in = (uint32_t)(t >> 32);
    }
  }
  // d = x - y; returns whether x < y (d is then x - y + 2^(32 G K)).
  static __device__ __forceinline__ bool minus(Num& d, const Num& x, const Num& y) {
    uint32_t br = 0;
    bool zero = true;
#pragma unroll
    for (int j = 0; j < K; ++j) {
      const uint64_t t = (uint64_t)x[j] - y[j] - br;
      d[j] = (uint32_t)t;
      br = (uint32_t)(t >> 32) & 1;
      zero &= d[j] == 0;
    }
    bool out;
    br = carry_in(br != 0, zero, out);
#pragma unroll
    for (int j = 0; j < K; ++j) {
      const uint64_t t = (uint64_t)d[j] - br;
      d[j] = (uint32_t)t;
      br = (uint32_t)(t >> 32) & 1;
    }
    return out;
  }
  static __device__ __forceinline__ bool equal(const Num& x, const Num& y) {
    bool same = true;
#pragma unroll
    for (int j = 0; j < K; ++j) same &= x[j] == y[j];
    const uint32_t b = __ballot_sync(kAllLanes, !same);
    const int lead = (threadIdx.x & 31) & ~(G - 1);
    return G == 32 ? b == 0 : ((b >> lead) & ((1u << (G & 31)) - 1)) == 0;
  }
  static __device__ __forceinline__ void copy(Num& r, const Num& x) {
#pragma unroll
    for (int j = 0; j < K; ++j) r[j] = x[j];
  }
  // x mod q for x < 2q
  static __device__ __forceinline__ void canon(Num& x, const Num& q) {
    Num d;
    if (!minus(d, x, q)) copy(x, d);
  }
  static __device__ __forceinline__ void dbl(Num& x, const Num& q) {  // 2x mod q for x < q
    uint32_t in = up(x[K - 1] >> 31);
#pragma unroll
    for (int j = 0; j < K; ++j) {
      const uint32_t o = x[j] >> 31;
      x[j] = (x[j] << 1) | in;
      in = o;
    }
    canon(x, q);
  }
  // One limb of Montgomery reduction of the number with the 64-bit limbs c, and
  // the limbs of another number added: c = (c + m q) / 2^32 + add with m = c (-q^-1)
  // mod 2^32.  qn: the lowest limb of q in the next lane; top: what c holds beyond
  // the last lane.  Every lane makes m itself, from lane 0's lowest limb, and
  // takes both the low half of its own products and the high half of those one
  // limb below, so the only exchange is the one that hands out that limb and
  // moves the limbs down.
  static __device__ __forceinline__ void reduce(uint64_t (&c)[K], const uint64_t (&add)[K], uint32_t top,
                                                const Num& q, uint32_t qn, uint32_t qinv) {
    const uint32_t t = __shfl_sync(kAllLanes, (uint32_t)c[0], 0, G);
    const uint32_t next = __shfl_down_sync(kAllLanes, (uint32_t)c[0], 1, G);
    const uint32_t m = t * qinv;
    uint64_t d[K];
#pragma unroll
    for (int j = 0; j < K; ++j)
      d[j] = (c[j] >> 32) + (j + 1 < K ? (uint32_t)c[j + 1] : sub() == G - 1 ? top : next) + add[j];
    d[0] += sub() == 0 && t != 0;  // t + (m q mod 2^32) is 0 or 2^32
#pragma unroll
    for (int j = 0; j < K; ++j) {
      const uint32_t hi = __umulhi(q[j], m), lo = (j + 1 < K ? q[j + 1] : qn) * m;
      c[j] = d[j] + hi + lo;
    }
  }
  // z = x v limb by limb (64-bit limbs); xb: the highest limb of x in the lane below
  static __device__ __forceinline__ void times(uint64_t (&z)[K], const Num& x, uint32_t xb, uint32_t v) {
#pragma unroll
    for (int j = 0; j < K; ++j) z[j] = (uint64_t)(x[j] * v) + __umulhi(j ? x[j - 1] : xb, v);
  }
  // x = x y / R mod q below 2q, R = 2^(32 K rl), for x, y < 2q
  static __device__ __forceinline__ void mul(Num& x, const Num& y, const Num& q, uint32_t qn, uint32_t qinv, int rl) {
    const uint32_t xb = up(x[K - 1]);
    uint64_t c[K], z[K];
    uint32_t v = __shfl_sync(kAllLanes, y[0], 0, G);
    times(c, x, xb, v);
    for (int l = 0; l < rl; ++l) {
#pragma unroll
      for (int j = 0; j < K; ++j) {
        const uint32_t top = __umulhi(x[K - 1], v);
        v = __shfl_sync(kAllLanes, y[j + 1 < K ? j + 1 : 0], j + 1 < K ? l : l + 1, G);
        if (j + 1 == K && l + 1 == rl) v = 0;  // past y
        times(z, x, xb, v);
        reduce(c, z, top, q, qn, qinv);
      }
    }
    settle(x, c);
  }
  // x = x 2^(s - 32) mod q below 2q, 0 <= s < 32, for x < 2q
  static __device__ __forceinline__ void shift(Num& x, uint32_t s, const Num& q, uint32_t qn, uint32_t qinv) {
    uint64_t c[K], z[K];
#pragma unroll
    for (int j = 0; j < K; ++j) {
      c[j] = (uint64_t)x[j] << s;
      z[j] = 0;
    }
    reduce(c, z, 0, q, qn, qinv);
    settle(x, c);
  }
};

// What a test of q needs: its limbs (in shared memory too, for the exponent's
// bits), -q^-1 mod 2^32, R mod q.
template <int G, int K>
struct BigMod {
  typedef Big<G, K> B;
  typename B::Num q, one;
  uint32_t qn, qinv;  // q's lowest limb in the next lane; -q^-1 mod 2^32
  int bits, s, rl;  // bit length of q, q - 1 = d 2^s, lanes of R

  // q = n - p; words: this group's q in shared memory (G K words)
  __device__ __forceinline__ BigMod(const BigArgs& a, uint32_t p, uint32_t* words) : rl((int)a.rl) {
    typename B::Num n, pn, z;
#pragma unroll
    for (int j = 0; j < K; ++j) {
      const uint32_t i = B::sub() * K + j;
      n[j] = i < a.nl ? a.n[i] : 0;
      pn[j] = i == 0 ? p : 0;
    }
    B::minus(q, n, pn);
    qn = __shfl_down_sync(kAllLanes, q[0], 1, G);
    if (B::sub() == G - 1) qn = 0;
    __syncwarp();
#pragma unroll
    for (int j = 0; j < K; ++j) words[B::sub() * K + j] = q[j];
    __syncwarp();
    uint32_t x = words[0];
    for (int i = 0; i < 4; ++i) x *= 2u - words[0] * x;
    qinv = 0u - x;
    int top = (int)a.nl - 1;
    while (words[top] == 0) --top;
    bits = 32 * top + 32 - __clz(words[top]);
    uint32_t low = words[0] & ~1u;
    int w = 0;
    while (low == 0) low = words[++w];
    s = 32 * w + __ffs(low) - 1;
    // R mod q: 2^bits - q, doubled up to R
#pragma unroll
    for (int j = 0; j < K; ++j) {
      const int i = B::sub() * K + j;
      z[j] = i == bits / 32 ? 1u << (bits & 31) : 0;
    }
    B::minus(one, z, q);
    // (the groups of a warp may differ by a bit: they run together)
    const int dbls = 32 * K * rl - bits;
    const int most = (int)__reduce_max_sync(kAllLanes, (uint32_t)dbls);
#pragma unroll 1
    for (int i = 0; i < most; ++i) {
      B::copy(z, one);
      B::dbl(z, q);
      if (i < dbls) B::copy(one, z);
    }
  }
  // The strong test's verdict from x = a^d (in Montgomery form, below 2q).
  __device__ __forceinline__ bool verdict(typename B::Num& x, int smax) const {
    typename B::Num mone, y;
    B::minus(mone, q, one);
    B::copy(y, x);
    B::canon(y, q);
    bool ok = B::equal(y, one) | B::equal(y, mone);
#pragma unroll 1
    for (int i = 1; i < smax; ++i) {
      B::copy(y, x);
      B::mul(x, y, q, qn, qinv, rl);
      B::copy(y, x);
      B::canon(y, q);
      ok |= B::equal(y, mone) && i < s;
    }
    return ok;
  }
};

// bits [b, b + w) of the number in words, w <= 8, b + w <= 32 * its words + 24
__device__ __forceinline__ uint32_t bits_at(const uint32_t* words, int nwords, int b, int w) {
  const int i = b >> 5;
  const uint32_t lo = words[i], hi = i + 1 < nwords ? words[i + 1] : 0;
  return __funnelshift_r(lo, hi, b & 31) & ((1u << w) - 1);
}

constexpr int kBigThreads = 64;
// Up to 32 limbs (K = 1) the other bases of the first survivors run beside base
// 2, in CTAs of the same launch: at 512 bits 85% of the n have their first prime
// among 32 (n of 512 bits 0.81 -> 0.53 ms, of 96 0.11 -> 0.086, of 1024 3.44 -> 3.38;
// longer n find it there less often than not, and their tests fill the lanes).
constexpr uint32_t kBigSpec = 32;
constexpr uint32_t kSpecCtas = kBigSpec * 11 / (kBigThreads / 32);

// The strong test of q = n - p to `base` by one warp.  Four exponent bits at a time,
// the powers base^0 .. base^15 in shared memory.
template <int G, int K>
struct BasesShared {
  uint32_t q[G * K], all[32 / G][G * K];
  uint32_t pow[16][32 * K];
};
template <int G, int K>
__device__ __forceinline__ bool big_strong(const BigArgs& a, uint32_t p, uint32_t base, BasesShared<G, K>& sm) {
  typedef Big<G, K> B;
  const uint32_t lane = threadIdx.x & 31;
  const BigMod<G, K> M(a, p, sm.all[lane / G]);  // every group of the warp holds the same q
  if (lane < G)
    for (int j = 0; j < K; ++j) sm.q[lane * K + j] = M.q[j];
  typename B::Num x, y, b;
  // base in Montgomery form, from the base's bits
#pragma unroll
  for (int j = 0; j < K; ++j) b[j] = 0;
  for (int k = 5; k >= 0; --k) {
    B::dbl(b, M.q);
    if ((base >> k) & 1u) {  // b + one mod q
      uint64_t c[K];
#pragma unroll
      for (int j = 0; j < K; ++j) c[j] = (uint64_t)b[j] + M.one[j];
      B::settle(b, c);
      B::canon(b, M.q);
    }
  }
  B::copy(x, M.one);
  for (int k = 0; k < 16; ++k) {
#pragma unroll
    for (int j = 0; j < K; ++j) sm.pow[k][lane * K + j] = x[j];
    B::mul(x, b, M.q, M.qn, M.qinv, M.rl);
  }
  __syncwarp();
  const int dbits = M.bits - M.s;
  int pos = (dbits - 1) / 4 * 4;  // the lowest bit of the top digit
  const auto load = [&](uint32_t d) {
#pragma unroll
    for (int j = 0; j < K; ++j) y[j] = sm.pow[d][lane * K + j];
  };
  load(bits_at(sm.q, G * K, M.s + pos, dbits - pos));
  B::copy(x, y);
#pragma unroll 1
  while (pos > 0) {
    pos -= 4;
#pragma unroll 1
    for (int k = 0; k < 4; ++k) {
      B::copy(y, x);
      B::mul(x, y, M.q, M.qn, M.qinv, M.rl);
    }
    load(bits_at(sm.q, G * K, M.s + pos, 4));
    B::mul(x, y, M.q, M.qn, M.qinv, M.rl);
  }
  return M.verdict(x, M.s);
}

// Phase 0: base 2 on every survivor, G lanes each.  The power is taken 5 bits
// at a time: five squarings take 2^e to 2^(32 e), and a shift by c with one limb
// of reduction to 2^(32 e + c - 32), so the digits c are those of d + 32 (1 + 32
// + ... + 32^(m-1)) in base 32: d's own, with one added from the second on and
// the carries passed up.  What is above the m digits (at most 33) is made by
// doublings of R mod q.
template <int G, int K>
__global__ void __launch_bounds__(kBigThreads) big_base2_kernel(const __grid_constant__ BigArgs a, uint32_t k0) {
  typedef Big<G, K> B;
  if constexpr (K == 1) {  // the first CTAs: a warp per base of the first survivors
    if (blockIdx.x < kSpecCtas) {
      __shared__ BasesShared<G, 1> sm[kBigThreads / 32];
      const uint32_t w = threadIdx.x >> 5, job = blockIdx.x * (kBigThreads / 32) + w;
      const uint32_t r = job / 11;
      if (r >= Survivors(a).total) return;
      if (!big_strong<G, 1>(a, a.primes[k0 + nth_survivor(a, r)], kBigBases[1 + job % 11], sm[w]) && (threadIdx.x & 31) == 0)
        atomicOr(a.specfail, 1u << r);
      return;
    }
  }
  const uint32_t cta = blockIdx.x - (K == 1 ? kSpecCtas : 0), ctas = gridDim.x - (K == 1 ? kSpecCtas : 0);
  constexpr int kGroups = kBigThreads / G;
  constexpr int kDigits = (32 * kBigMaxLimbs + 4) / 5;
  __shared__ uint32_t s_q[kGroups][G * K];
  __shared__ uint8_t s_dig[kGroups][K == 1 ? 32 * G / 5 + 1 : kDigits];
  const uint32_t gi = threadIdx.x / G;
  uint32_t* words = s_q[gi];
  uint8_t* dig = s_dig[gi];
  const uint32_t nsurv = Survivors(a).total, groups = ctas * kGroups;
  for (uint32_t t0 = cta * kGroups; t0 < nsurv; t0 += groups) {  // uniform in the CTA
    const uint32_t t = t0 + gi;
    const bool act = t < nsurv;  // a group past the end runs along on the last survivor
    const uint32_t i = nth_survivor(a, t);
    const BigMod<G, K> M(a, a.primes[k0 + i], words);
    if (act && B::sub() == 0) atomicAdd(a.mr_tests, 1ull);
    const int dbits = M.bits - M.s;
    const int m = dbits > 5 ? (dbits - 1) / 5 : 0;  // at least one bit stays above
    uint32_t e0 = 0;
    if (B::sub() == 0) {
      uint32_t carry = 0;
      for (int j = 0; j < m; ++j) {
        const uint32_t v = bits_at(words, G * K, M.s + 5 * j, 5) + (j > 0) + carry;
        dig[j] = (uint8_t)(v & 31);
        carry = v >> 5;
      }
      e0 = bits_at(words, G * K, M.s + 5 * m, dbits - 5 * m) + (m > 0) + carry;
    }
    __syncwarp();
    e0 = __shfl_sync(kAllLanes, e0, 0, G);
    const int mmax = (int)__reduce_max_sync(kAllLanes, (uint32_t)m);
    const uint32_t emax = __reduce_max_sync(kAllLanes, e0);
    typename B::Num x, y;
    B::copy(x, M.one);
    for (uint32_t j = 0; j < emax; ++j) {
      B::copy(y, x);
      B::dbl(y, M.q);
      if (j < e0) B::copy(x, y);
    }
#pragma unroll 1
    for (int j = mmax - 1; j >= 0; --j) {
#pragma unroll 1
      for (int k = 0; k < 5; ++k) {
        B::copy(y, x);
        B::mul(y, x, M.q, M.qn, M.qinv, M.rl);
        if (j < m) B::copy(x, y);
      }
      B::copy(y, x);
      B::shift(y, j < m ? dig[j] : 0, M.q, M.qn, M.qinv);
      if (j < m) B::copy(x, y);
    }
    const bool ok = M.verdict(x, (int)__reduce_max_sync(kAllLanes, (uint32_t)M.s));
    if (ok && act && B::sub() == 0) {
      a.pass[atomicAdd(a.npass, 1u)] = i;
      atomicMin(a.minpass, i);
    }
    __syncwarp();
  }
}

// Phase 1: bases 3, ..., 37 on one passer (i, or the smallest for ~0u), a warp per
// base; a failing base sets *fail.  A passer among the first kBigSpec survivors
// has been through them beside base 2.
template <int G, int K>
__global__ void __launch_bounds__(32) big_bases_kernel(const __grid_constant__ BigArgs a, uint32_t k0, uint32_t i) {
  __shared__ BasesShared<G, K> sm;
  if (i == 0xffffffffu) i = *a.minpass;
  if (i == 0xffffffffu) return;  // no candidate passed base 2
  if constexpr (K == 1) {
    const uint32_t r = Survivors(a).rank(i);
    if (r < kBigSpec) {
      if (blockIdx.x == 0 && threadIdx.x == 0 && (*a.specfail >> r & 1)) *a.fail = 1;
      return;
    }
  }
  const bool ok = big_strong<G, K>(a, a.primes[k0 + i], kBigBases[1 + blockIdx.x], sm);
  if (!ok && threadIdx.x == 0) atomicOr(a.fail, 1u);
}

cudaError_t launch_big_filter(const BigArgs& a, uint32_t k0, uint32_t kcount, cudaStream_t s) {
  big_filter_kernel<<<(kcount + 31) / 32, kFilterThreads, 0, s>>>(a, k0, kcount);
  return cudaGetLastError();
}

// Lanes and limbs per lane for R of `limbs` limbs (at most GB_BIG_MAX_LIMBS + 1).
static void big_shape(uint32_t limbs, int& G, int& K) {
  G = limbs <= 8 ? 8 : limbs <= 16 ? 16 : 32;
  K = limbs <= 32 ? 1 : limbs <= 64 ? 2 : limbs <= 96 ? 3 : limbs <= 128 ? 4 : 5;
}

uint32_t big_r_lanes(uint32_t limbs) {
  int G, K;
  big_shape(limbs, G, K);
  return (limbs + K - 1) / K;
}

template <typename F>
static cudaError_t with_big_shape(uint32_t limbs, F f) {
  int G, K;
  big_shape(limbs, G, K);
  if (G == 8) f(std::integral_constant<int, 8>{}, std::integral_constant<int, 1>{});
  else if (G == 16) f(std::integral_constant<int, 16>{}, std::integral_constant<int, 1>{});
  else if (K == 1) f(std::integral_constant<int, 32>{}, std::integral_constant<int, 1>{});
  else if (K == 2) f(std::integral_constant<int, 32>{}, std::integral_constant<int, 2>{});
  else if (K == 3) f(std::integral_constant<int, 32>{}, std::integral_constant<int, 3>{});
  else if (K == 4) f(std::integral_constant<int, 32>{}, std::integral_constant<int, 4>{});
  else f(std::integral_constant<int, 32>{}, std::integral_constant<int, 5>{});
  return cudaGetLastError();
}

cudaError_t launch_big_base2(const BigArgs& a, uint32_t k0, int grid, cudaStream_t s) {
  return with_big_shape(a.limbs, [&](auto g, auto k) {
    constexpr int K = decltype(k)::value;
    big_base2_kernel<decltype(g)::value, K><<<grid + (K == 1 ? kSpecCtas : 0), kBigThreads, 0, s>>>(a, k0);
  });
}

cudaError_t launch_big_bases(const BigArgs& a, uint32_t k0, uint32_t i, cudaStream_t s) {
  return with_big_shape(a.limbs, [&](auto g, auto k) {
    big_bases_kernel<decltype(g)::value, decltype(k)::value><<<11, 32, 0, s>>>(a, k0, i);
  });
}

}  // namespace gb
