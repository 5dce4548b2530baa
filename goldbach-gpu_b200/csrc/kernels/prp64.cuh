// prp64.cuh -- primality of odd 64-bit q on a warp (sm_100a): the base-2
// strong test of 32 lanes at once, and the extra strong Lucas test that
// makes a base-2 pass a proof.
//
// A q that passes the strong test to base 2 and the extra strong Lucas test
// (Q = 1, the first P >= 3 with (P^2 - 4 | q) = -1) is prime for every
// q < 2^64: the combination is the Baillie-PSW test (Baillie and Wagstaff,
// "Lucas pseudoprimes", Math. Comp. 35, 1980; extra strong Lucas: Grantham,
// "Frobenius pseudoprimes", Math. Comp. 70, 2001), and none of the
// 118,968,378 base-2 pseudoprimes below 2^64 that Feitsma enumerated passes
// the Lucas half.  It replaces the six other strong tests of the 7-base set
// (and of the reference's 12-base set, src/goldbach.cu:333-360), which cost
// 6 x 95 Montgomery products per prime, by 128.
//
// What bounds the tests is the multiplier: one IMAD.WIDE (32 x 32 + 64) takes
// the issue slots of about two 32-bit IMADs, and a product costs 8 of them
// whatever the form (measured on a B200, clocks per warp product at 16 warps
// per SM quarter: operand scanning with a final subtraction, mont_mul32 53.7;
// 64-bit halves from __umul64hi 57.7; 31-bit limbs without carries 50.1; the
// lazy form below 40.7).  So the work is cut elsewhere:
//   * the base-2 power is taken 5 exponent bits at a time: five squarings,
//     then one multiplication by 2^c as a shift and a one-limb reduction
//     (about a third of a product), where a 2-bit window needs a full
//     product every two bits and three table values in registers;
//   * moduli below 2^62 keep their residues in [0, 2n), so a product has no
//     final subtraction (mont_mul_lazy: 40.7 against 53.7 clocks).
#pragma once
#include <cstdint>

#include "../gb_device.cuh"

namespace gb {

constexpr uint64_t kLazyTop = 1ull << 62;  // moduli below it may take the lazy form

// a * b * 2^-64 mod n in [0, 2n) for a, b in [0, 2n), n < 2^62: the high
// limbs stay below 2^31, so the middle column fits 64 bits and the sum of
// the product (< 4n^2) and the reduction (< 2^64 n) fits 128.  ni = -n^-1
// mod 2^32.
__device__ __forceinline__ uint64_t mont_mul_lazy(uint64_t a, uint64_t b, uint64_t n, uint32_t ni) {
  const uint32_t a0 = (uint32_t)a, a1 = (uint32_t)(a >> 32);
  const uint32_t b0 = (uint32_t)b, b1 = (uint32_t)(b >> 32);
  const uint64_t c0 = (uint64_t)a0 * b0;
  const uint64_t c1 = (uint64_t)a0 * b1 + (uint64_t)a1 * b0;
  const uint64_t c2 = (uint64_t)a1 * b1;
  uint32_t t0 = (uint32_t)c0, t1 = (uint32_t)(c0 >> 32), t2 = (uint32_t)c2, t3 = (uint32_t)(c2 >> 32);
  asm("{\n\t"
      ".reg .u32 m, z;\n\t"
      "add.cc.u32 %1, %1, %4;\n\t"
      "addc.cc.u32 %2, %2, %5;\n\t"
      "addc.u32 %3, %3, 0;\n\t"
      "mul.lo.u32 m, %0, %8;\n\t"
      "mad.lo.cc.u32 z, m, %6, %0;\n\t"
      "madc.hi.cc.u32 %1, m, %6, %1;\n\t"
      "addc.cc.u32 %2, %2, 0;\n\t"
      "addc.u32 %3, %3, 0;\n\t"
      "mad.lo.cc.u32 %1, m, %7, %1;\n\t"
      "madc.hi.cc.u32 %2, m, %7, %2;\n\t"
      "addc.u32 %3, %3, 0;\n\t"
      "mul.lo.u32 m, %1, %8;\n\t"
      "mad.lo.cc.u32 z, m, %6, %1;\n\t"
      "madc.hi.cc.u32 %2, m, %6, %2;\n\t"
      "addc.u32 %3, %3, 0;\n\t"
      "mad.lo.cc.u32 %2, m, %7, %2;\n\t"
      "madc.hi.u32 %3, m, %7, %3;\n\t"
      "}"
      : "+r"(t0), "+r"(t1), "+r"(t2), "+r"(t3)
      : "r"((uint32_t)c1), "r"((uint32_t)(c1 >> 32)), "r"((uint32_t)n), "r"((uint32_t)(n >> 32)), "r"(ni));
  return ((uint64_t)t3 << 32) | t2;
}

// Residues mod n in Montgomery form (R = 2^64): in [0, n) for any odd n
// (LAZY false), in [0, 2n) for n < 2^62 (LAZY true).
template <bool LAZY>
struct Ring64 {
  uint64_t n;
  uint32_t ni;  // -n^-1 mod 2^32
  __device__ __forceinline__ uint64_t mul(uint64_t a, uint64_t b) const {
    return LAZY ? mont_mul_lazy(a, b, n, ni) : mont_mul32(a, b, n, ni);
  }
  // x 2^(c - 32) mod n, 0 <= c < 32: the 96-bit x 2^c and one limb of
  // Montgomery reduction.  Lazy: (2n 2^31 + 2^32 n) / 2^32 = 2n bounds it;
  // else the difference of the high parts lies in (-n, n / 2).
  __device__ __forceinline__ uint64_t shift(uint64_t x, uint32_t c) const {
    const uint32_t x0 = (uint32_t)x, x1 = (uint32_t)(x >> 32);
    const uint32_t n0 = (uint32_t)n, n1 = (uint32_t)(n >> 32);
    const uint32_t t0 = x0 << c, t1 = __funnelshift_l(x0, x1, c), t2 = __funnelshift_l(x1, 0u, c);
    if (LAZY) {
      const uint32_t m = t0 * ni;
      uint32_t r1 = t1, r2 = t2;
      asm("{\n\t"
          ".reg .u32 z;\n\t"
          "mad.lo.cc.u32 z, %2, %3, %5;\n\t"
          "madc.hi.cc.u32 %0, %2, %3, %0;\n\t"
          "addc.u32 %1, %1, 0;\n\t"
          "mad.lo.cc.u32 %0, %2, %4, %0;\n\t"
          "madc.hi.u32 %1, %2, %4, %1;\n\t"
          "}"
          : "+r"(r1), "+r"(r2)
          : "r"(m), "r"(n0), "r"(n1), "r"(t0));
      return ((uint64_t)r2 << 32) | r1;
    }
    const uint32_t m = t0 * (0u - ni);
    const uint64_t g = (uint64_t)m * n1 + __umulhi(m, n0);
    const uint64_t t = ((uint64_t)t2 << 32) | t1;
    return t < g ? t - g + n : t - g;
  }
  __device__ __forceinline__ uint64_t dbl(uint64_t x) const {  // keeps the bound of its argument
    const uint64_t s = x + x, b = LAZY ? 2 * n : n;
    return (!LAZY && s < x) || s >= b ? s - b : s;
  }
  __device__ __forceinline__ uint64_t sub(uint64_t x, uint64_t y) const {  // y in [0, n)
    const uint64_t d = x - y;
    return x < y ? d + (LAZY ? 2 * n : n) : d;
  }
  __device__ __forceinline__ uint64_t canon(uint64_t x) const { return LAZY && x >= n ? x - n : x; }
};

// R mod n for odd n >= 3 without a division: 2^(k+1) - n for the top bit k
// of n, doubled up to 2^64 (not at all for n >= 2^63).
__device__ __forceinline__ uint64_t mont_one(uint64_t n) {
  const int k = 63 - __clzll(n);
  uint64_t x = k == 63 ? 0 - n : (2ull << k) - n;
  for (int j = k + 1; j < 64; ++j) x = mod_dbl(x, n);
  return x;
}

// -n^-1 mod 2^32 by Newton steps.
__device__ __forceinline__ uint32_t neg_inv32(uint32_t n) {
  uint32_t x = n;  // 3 correct bits
#pragma unroll
  for (int i = 0; i < 4; ++i) x *= 2u - n * x;
  return 0u - x;
}

// Strong probable-prime test to base 2 of every lane's odd n >= 3 (lanes with
// act false run along; any odd n >= 3 will do there).  All 32 lanes call it.
//
// With X = 2^(e + 64) mod n (2^e in Montgomery form), five squarings take e
// to 32 e and shift(X, c) takes it to e + c - 32: a step is e -> 32 e + c -
// 32.  From e0 and digits c, m steps reach 2^d when e0 32^m + sum of c 32^i
// is D = d + 32 (1 + 32 + ... + 32^(m-1)), so the digits are D's in base 32
// and e0 = D >> 5m is made by doublings of 1.  m is the same for the whole
// warp, 4 bits short of the longest exponent: e0 <= 17, and D < 2^64 because
// m <= 12 and d < 2^63.
template <bool LAZY>
__device__ __forceinline__ bool sprp2_warp(uint64_t n, bool act) {
  constexpr uint32_t kAll = 0xffffffffu;
  const Ring64<LAZY> r{n, neg_inv32((uint32_t)n)};
  const uint64_t one = mont_one(n);
  uint64_t d = n - 1;
  const int s = __ffsll((long long)d) - 1;
  d >>= s;
  const int bits = (int)__reduce_max_sync(kAll, act ? 64u - __clzll(d) : 0u);
  const int m = bits > 4 ? bits / 5 : 0;  // ceil((bits - 4) / 5)
  constexpr uint64_t kRep = 0x0084210842108421ull;  // sum of 32^i, i < 12
  const uint64_t D = d + ((kRep & ((1ull << (5 * m)) - 1)) << 5);
  const uint32_t e0 = (uint32_t)(D >> (5 * m));
  const uint32_t emax = __reduce_max_sync(kAll, act ? e0 : 0u);
  uint64_t x = one;
  for (uint32_t j = 0; j < emax; ++j) x = j < e0 ? r.dbl(x) : x;
#pragma unroll 1
  for (int i = 5 * (m - 1); i >= 0; i -= 5) {
#pragma unroll
    for (int j = 0; j < 5; ++j) x = r.mul(x, x);
    x = r.shift(x, (uint32_t)(D >> i) & 31u);
  }
  const uint64_t mone = n - one;
  uint64_t y = r.canon(x);
  bool ok = y == one || y == mone;
  const int S = (int)__reduce_max_sync(kAll, act ? (uint32_t)s : 0u);
#pragma unroll 1
  for (int i = 1; i < S; ++i) {
    x = r.mul(x, x);
    y = r.canon(x);
    ok |= i < s && y == mone;
  }
  return ok;
}

// Jacobi symbol (a | u) for odd u, a < u.
__device__ __forceinline__ int jacobi32(uint32_t a, uint32_t u) {
  int j = 1;
  while (a) {
    const int z = __ffs((int)a) - 1;
    a >>= z;
    if ((z & 1) && ((u & 7) == 3 || (u & 7) == 5)) j = -j;
    if ((a & 3) == 3 && (u & 3) == 3) j = -j;
    const uint32_t t = u % a;
    u = a;
    a = t;
  }
  return u == 1 ? j : 0;
}

// (l | n) for an odd prime l < 64 from n mod l: qr holds the squares mod l,
// and reciprocity flips the sign when both are 3 mod 4.  False: -1.
__device__ __forceinline__ bool residue_plus(uint32_t r, uint32_t l, uint64_t qr, bool n3mod4) {
  return (((qr >> r) & 1) != 0) != ((l & 3) == 3 && n3mod4);
}
struct LucasPrimes {  // the primes 11, 13, ..., 61 and the squares mod each
  uint32_t l[14];
  uint64_t qr[14];
  constexpr LucasPrimes() : l(), qr() {
    int c = 0;
    for (uint32_t v = 11; c < 14; v += 2) {
      if (v % 3 == 0 || v % 5 == 0 || v % 7 == 0) continue;
      l[c] = v;
      for (uint32_t x = 1; x < v; ++x) qr[c] |= 1ull << (x * x % v);
      ++c;
    }
  }
};
__device__ __constant__ const LucasPrimes kLucasPrimes{};

// The extra strong Lucas test's P: the smallest P >= 3 with (P^2 - 4 | n) =
// -1.  A prime l first divides P^2 - 4 = (P - 2)(P + 2) at P = l - 2, beside
// smaller primes only (3 at P = 4; 2, to an odd power, at P = 6), so P comes
// from the first of 5, 3, 7, 2, 11, 13, ... whose symbol is -1; past 61
// (one n in 2^18) the symbols of P^2 - 4 itself are tried in order.  0 when
// one of those numbers shares a factor with n (composite: n > 2^13; a
// square's search ends there too, at the latest at its root).
__device__ __forceinline__ uint32_t lucas_param(uint64_t n) {
  const bool n3mod4 = (n & 3) == 3;
  // residues from n's halves: the moduli are small, so the sums fit 32 bits
  const uint32_t hi = (uint32_t)(n >> 32), lo = (uint32_t)n;
  const uint32_t r105 = ((hi % 105u) * (4294967296ull % 105u) + lo % 105u) % 105u;
  const uint32_t r5 = r105 % 5, r3 = r105 % 3, r7 = r105 % 7, r8 = lo & 7;
  if (r5 == 2 || r5 == 3) return 3;
  if (r5 == 0 || r3 == 0) return 0;
  if (!residue_plus(r3, 3, 0x2, n3mod4)) return 4;
  if (r7 == 0) return 0;
  if (!residue_plus(r7, 7, 0x16, n3mod4)) return 5;
  if (r8 == 3 || r8 == 5) return 6;
#pragma unroll 1
  for (int i = 0; i < 14; ++i) {
    const uint32_t l = kLucasPrimes.l[i];
    const uint32_t r = ((hi % l) * ((0xffffffffu % l + 1) % l) + lo % l) % l;
    if (r == 0) return 0;
    if (!residue_plus(r, l, kLucasPrimes.qr[i], n3mod4)) return l - 2;
  }
#pragma unroll 1
  for (uint32_t P = 60; P < 65536; ++P) {
    uint32_t u = P * P - 4;
    const int z = __ffs((int)u) - 1;
    u >>= z;
    int j = (z & 1) && (r8 == 3 || r8 == 5) ? -1 : 1;
    if ((u & 3) == 3 && n3mod4) j = -j;
    j *= jacobi32((uint32_t)(n % u), u);
    if (j < 0) return P;
    if (j == 0) return 0;
  }
  return 0;
}

// A modulus' constants for the Lucas ladder.
template <bool LAZY>
struct LucasRing : Ring64<LAZY> {
  uint64_t two, p;  // 2 and P in Montgomery form
  uint32_t P;
  __device__ __forceinline__ LucasRing(uint64_t n, bool act) : Ring64<LAZY>{n, neg_inv32((uint32_t)n)} {
    const uint64_t one = mont_one(n);
    two = mod_dbl(one, n);
    P = act ? lucas_param(n) : 3u;
    p = 0;
    for (int b = 31 - __clz(P | 1u); b >= 0; --b) {
      p = mod_dbl(p, n);
      if ((P >> b) & 1u) {
        const uint64_t t = p + one;
        p = t < p || t >= n ? t - n : t;
      }
    }
  }
  // the verdict from V_d and V_{d+1}, n + 1 = d 2^s; S: the warp's largest s
  __device__ __forceinline__ bool verdict(uint64_t v, uint64_t w, int s, int S) const {
    uint64_t x = this->canon(v);
    const uint64_t y = this->canon(w), n = this->n;
    bool ok = (x == two && y == p) || (x == n - two && y == n - p);
#pragma unroll 1
    for (int i = 0; i + 1 < S; ++i) {
      ok |= i + 1 < s && x == 0;
      v = this->sub(this->mul(v, v), two);
      x = this->canon(v);
    }
    return ok && P != 0;
  }
};

// Extra strong Lucas test of every lane's odd n > 2^13, n < 2^64 - 1 (lanes
// with act false run along).  All 32 lanes call it.  With n + 1 = d 2^s: V_d =
// +-2 and U_d = 0 (that is V_{d+1} = +-P), or V_{2^r d} = 0 for some r < s - 1.
// The ladder keeps (V_k, V_{k+1}), two independent products per bit; from k =
// 0, (2, P), leading zero bits change nothing, so the warp runs its longest d.
template <bool LAZY>
__device__ __forceinline__ bool lucas_warp(uint64_t n, bool act) {
  constexpr uint32_t kAll = 0xffffffffu;
  const LucasRing<LAZY> r(n, act);
  uint64_t d = n + 1;
  const int s = __ffsll((long long)d) - 1;
  d >>= s & 63;
  const int top = (int)__reduce_max_sync(kAll, act ? 63u - __clzll(d | 1) : 0u);
  uint64_t v = r.two, w = r.p;
#pragma unroll 1
  for (int i = top; i >= 0; --i) {
    const bool b = (d >> i) & 1;
    const uint64_t t = b ? w : v;
    const uint64_t m = r.sub(r.mul(v, w), r.p);
    const uint64_t q = r.sub(r.mul(t, t), r.two);
    v = b ? m : q;
    w = b ? q : m;
  }
  return r.verdict(v, w, s, (int)__reduce_max_sync(kAll, act ? (uint32_t)s : 0u));
}

// The same with a pair of lanes per n (both lanes of a pair pass the same n
// and act, and get the verdict): the even lane holds V_k, the odd one
// V_{k+1}, and each takes one product per bit.  The ladder's latency is what a
// small batch waits for, and two products in one lane do not overlap fully.
template <bool LAZY>
__device__ __forceinline__ bool lucas_pair(uint64_t n, bool act) {
  constexpr uint32_t kAll = 0xffffffffu;
  const LucasRing<LAZY> r(n, act);
  const bool odd = threadIdx.x & 1;
  uint64_t d = n + 1;
  const int s = __ffsll((long long)d) - 1;
  d >>= s & 63;
  const int top = (int)__reduce_max_sync(kAll, act ? 63u - __clzll(d | 1) : 0u);
  uint64_t x = odd ? r.p : r.two;
#pragma unroll 1
  for (int i = top; i >= 0; --i) {
    // V_k V_{k+1} - P, or this lane's own square - 2
    const bool cross = (((d >> i) & 1) != 0) != odd;
    const uint64_t y = __shfl_xor_sync(kAll, x, 1);
    x = r.sub(r.mul(x, cross ? y : x), cross ? r.p : r.two);
  }
  const uint64_t y = __shfl_xor_sync(kAll, x, 1);
  return r.verdict(odd ? y : x, odd ? x : y, s, (int)__reduce_max_sync(kAll, act ? (uint32_t)s : 0u));
}

// The whole warp's tests, in the lazy form when every active lane's n allows
// it.
__device__ __forceinline__ bool sprp2_any(uint64_t n, bool act) {
  return __any_sync(0xffffffffu, act && n >= kLazyTop) ? sprp2_warp<false>(n, act) : sprp2_warp<true>(act ? n : 3, act);
}
__device__ __forceinline__ bool lucas_any(uint64_t n, bool act) {
  return __any_sync(0xffffffffu, act && n >= kLazyTop) ? lucas_warp<false>(n, act) : lucas_warp<true>(act ? n : 3, act);
}
__device__ __forceinline__ bool lucas_pair_any(uint64_t n, bool act) {
  return __any_sync(0xffffffffu, act && n >= kLazyTop) ? lucas_pair<false>(n, act) : lucas_pair<true>(act ? n : 3, act);
}

}  // namespace gb
