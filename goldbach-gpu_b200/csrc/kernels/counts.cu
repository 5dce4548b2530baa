// counts.cu -- Goldbach partition counts c(n) on the GPU.
//
// c(n) = #{p <= n/2 : p and n - p prime}, the reference's goldbach_count
// (src/cpu_goldbach.cpp:29-36, a scalar scan over a byte table on the CPU;
// "partition counting c(n) at scale" is its open roadmap item,
// RESULTS.md:169).  The primes are split by residue: for a modulus M (2, 30 or
// 210) and a residue a prime to it, C_a is the bitset of the primes M k + a.
// With n = M t + r, p = a and q = b (mod M) need a + b = r (mod M), so
//     c(n) = sum over the pairs {a, b} of sum_k C_a[k] C_b[s - k]
//            + #{p | M : p <= n/2, n - p prime},     s = t - (a + b - r) / M,
// k over 0 .. s, or 0 .. s/2 for a = b.  A larger M leaves fewer pairs to test
// (n/4 of them per n for M = 2, 0.071 and 0.052 n on average for 30 and 210; 6,
// with 0.11, is never the cheapest) but takes more n to fill the groups of 32 n of one residue below; the
// host picks the M with the least work (counts_impl).
//
// A warp takes one pair {a, b}, 32 consecutive n of one residue (s0 .. s0 + 31)
// and a slice of C_a's words.  For word w the 32 bits C_b[s0 + d - 32w - i] (i =
// 0..31) of every d come from one 64-bit window of C_b read at s0 - 32w - 31,
// bit-reversed once, then funnel-shifted by d: an AND tests 32 pairs.  Seven
// words at a time go through four full adders (two three-input logic
// operations each), so three population counts serve seven words: a count
// takes 8 clocks of its pipe per warp and bound the loop before (9.5 clocks a
// word).  Now the ALU pipe does (shift, AND and adders, 3.1 instructions a word at
// 2 clocks).  Lanes accumulate 32 counters each, reduced across the warp by a
// transposing butterfly (lane d ends with the total of n's d-th).
// 4096 n near 1e9: 8.7 -> 2.4 ms, of which the sieve 0.3 and the classes 0.1
// (one CTA per SM at 255 registers 2.75, two 2.47, sums on the multiplier 2.38,
// three CTAs with spills 2.36; shifts on the multiplier too 2.5 to 2.7).
#include <cuda_runtime.h>

#include <cstdint>

#include "../gb_internal.h"

namespace gb {

constexpr int kCountThreads = 256;
constexpr int kCountWarps = kCountThreads / 32;

// full adder of three words: weight-1 and weight-2 bits
__device__ __forceinline__ void full_add(uint32_t a, uint32_t b, uint32_t c, uint32_t& s, uint32_t& t) {
  s = a ^ b ^ c;
  t = (a & b) | (a & c) | (b & c);
}

__global__ void __launch_bounds__(kCountThreads, 2) counts_kernel(const __grid_constant__ CountArgs a) {
  const int lane = threadIdx.x & 31;
  uint64_t task = (uint64_t)blockIdx.x * kCountWarps + (threadIdx.x >> 5);
  const uint64_t sp = task % a.splits;
  task /= a.splits;
  const uint64_t g = task % a.groups;
  if (task / a.groups >= a.npairs) return;  // warp-uniform, like the exits below
  const CountPair pr = a.npairs == 1 ? a.first : a.pairs[task / a.groups];
  if (g * 32 >= pr.count) return;
  const int64_t s0 = (int64_t)(pr.s0 + 32 * g);
  const int64_t last = pr.half ? (s0 + 31) / 2 : s0 + 31;  // largest k of any d
  const uint64_t nw = (uint64_t)last / 32 + 1;
  const uint64_t w_lo = sp * a.wps;
  if (w_lo >= nw) return;
  const uint64_t w_hi = w_lo + a.wps < nw ? w_lo + a.wps : nw;
  // words whose 32 k all count for every d (the padding clears k > s for a != b)
  const uint64_t full = !pr.half ? nw : s0 / 2 >= 31 ? (s0 / 2 - 31) / 32 + 1 : 0;
  const uint32_t* __restrict__ A = a.classes + pr.a * a.stride;
  // word w's window of C_b: 64 bits from s0 - 31 - 32w on (>= -63: the padding)
  const int64_t base = s0 - 31;
  const uint32_t sh = (uint32_t)base & 31u;
  const uint32_t* __restrict__ Bw = a.classes + pr.b * a.stride + (base >> 5);
  uint32_t acc[32];
#pragma unroll
  for (int d = 0; d < 32; ++d) acc[d] = 0;
  uint64_t w = w_lo + lane;
  const uint64_t f_hi = w_hi < full ? w_hi : full;
#pragma unroll 1
  for (; w + 6 * 32 < f_hi; w += 7 * 32) {
    uint32_t bw[7], rl[7], rh[7];
#pragma unroll
    for (int i = 0; i < 7; ++i) {
      const uint64_t wi = w + 32 * i;
      bw[i] = A[wi];
      const uint32_t* x = Bw - (int64_t)wi;
      const uint32_t x0 = x[0], x1 = x[1], x2 = x[2];
      rl[i] = __brev(__funnelshift_r(x1, x2, sh));
      rh[i] = __brev(__funnelshift_r(x0, x1, sh));
    }
#pragma unroll
    for (int d = 0; d < 32; ++d) {
      uint32_t x[7];
#pragma unroll
      for (int i = 0; i < 7; ++i)
        x[i] = bw[i] & __funnelshift_rc(rl[i], rh[i], 32 - d);
      uint32_t s1, s2, s3, s4, c1, c2, c3, c4;
      full_add(x[0], x[1], x[2], s1, c1);
      full_add(x[3], x[4], x[5], s2, c2);
      full_add(s1, s2, x[6], s3, c3);
      full_add(c1, c2, c3, s4, c4);
      // sums by multiply-adds: the logic and shifts already fill the ALU pipe
      acc[d] = __popc(s3) * a.one + acc[d];
      acc[d] = __popc(s4) * (2 * a.one) + acc[d];
      acc[d] = __popc(c4) * (4 * a.one) + acc[d];
    }
  }
#pragma unroll 1
  for (; w < w_hi; w += 32) {
    const uint32_t bw = A[w];
    const uint32_t* x = Bw - (int64_t)w;
    const uint32_t x0 = x[0], x1 = x[1], x2 = x[2];
    const uint32_t rl = __brev(__funnelshift_r(x1, x2, sh));
    const uint32_t rh = __brev(__funnelshift_r(x0, x1, sh));
#pragma unroll
    for (int d = 0; d < 32; ++d) {
      uint32_t mk = 0xffffffffu;
      if (w >= full) {  // a = b: only k <= floor((s0 + d) / 2) count
        const int64_t lim = (s0 + d) / 2 - 32 * (int64_t)w;
        mk = s0 + d < 0 || lim < 0 ? 0u : lim >= 31 ? 0xffffffffu : (2u << lim) - 1u;
      }
      acc[d] += __popc(bw & mk & __funnelshift_rc(rl, rh, 32 - d));
    }
  }
  // transposing butterfly: after the step of width k a lane keeps the half of
  // its counters selected by its lane bit k and adds the partner's copy
#pragma unroll
  for (int k = 16; k >= 1; k >>= 1) {
    const bool up = lane & k;
#pragma unroll
    for (int j = 0; j < k; ++j) {
      const uint32_t keep = up ? acc[j + k] : acc[j];
      const uint32_t give = up ? acc[j] : acc[j + k];
      acc[j] = keep + __shfl_xor_sync(0xffffffffu, give, k);
    }
  }
  const uint64_t j = g * 32 + lane;
  if (j < pr.count && acc[0]) atomicAdd(&a.out[pr.out + j * (a.modulus / 2)], (unsigned long long)acc[0]);
}

// The primes dividing M, which no class holds: out[j] = #{p | M : p <= n/2, n - p
// prime} (p = 2 only for n = 4).  odd: bit i <-> 2i + 1 prime, nodd words; the
// padding around them, which no other word of the call lies in, is cleared on the
// way (a memset before and one behind the sieve cost a small call 4 us of its 44).
__global__ void counts_small_kernel(uint32_t* odd, uint64_t nodd, uint64_t start, uint64_t count, uint32_t modulus,
                                    unsigned long long* __restrict__ out) {
  const uint64_t j = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (j < 8) odd[j < 2 ? (int64_t)j - 2 : (int64_t)(nodd + j - 2)] = 0;
  if (j >= count) return;
  const uint64_t n = start + 2 * j;
  uint32_t c = n == 4;
  for (uint32_t p = 3; p <= 7; p += 2)
    if (modulus % p == 0 && 2ull * p <= n) {
      const uint64_t i = (n - p) / 2;  // n - p = 2i + 1
      c += (odd[i >> 5] >> (i & 31)) & 1u;
    }
  out[j] = c;
}

// Class bitsets from the odd-only one.  A thread builds word W of every class:
// its 32 values of k span 16 M consecutive odd numbers, M / 2 words.
constexpr int kGatherThreads = 64;
template <int M>
__global__ void __launch_bounds__(kGatherThreads) gather_kernel(const uint32_t* __restrict__ odd, uint64_t nodd,
                                                                uint32_t* __restrict__ classes, uint64_t stride,
                                                                uint64_t nwords) {
  constexpr int H = M / 2;  // odd numbers, and words of 32, per k and per word of the classes
  __shared__ uint32_t tile[kGatherThreads * H];
  const uint64_t W0 = (uint64_t)blockIdx.x * kGatherThreads;
  for (uint32_t i = threadIdx.x; i < kGatherThreads * H; i += kGatherThreads) {
    const uint64_t w = W0 * H + i;
    tile[i] = w < nodd ? odd[w] : 0;
  }
  __syncthreads();
  const uint64_t W = W0 + threadIdx.x;
  if (W >= nwords) return;
  const uint32_t* t = tile + threadIdx.x * H;
  int c = 0;
  for (int a = 1; a < M; a += 2) {
    if (a % 3 == 0 || a % 5 == 0 || (M % 7 == 0 && a % 7 == 0)) continue;
    uint32_t v = 0;
#pragma unroll 8
    for (int b = 0; b < 32; ++b) {
      const int i = H * b + a / 2;  // odd number 2i + 1 = M b + a
      v |= ((t[i >> 5] >> (i & 31)) & 1u) << b;
    }
    classes[c++ * stride + W] = v;
  }
}

cudaError_t launch_count_classes(const uint32_t* odd, uint64_t nodd, uint32_t modulus, uint32_t* classes,
                                 uint64_t stride, uint64_t nwords, cudaStream_t s) {
  const uint64_t blocks = (nwords + kGatherThreads - 1) / kGatherThreads;
  if (blocks > 0x7fffffffull) return cudaErrorInvalidValue;
  switch (modulus) {
    case 30: gather_kernel<30><<<(unsigned)blocks, kGatherThreads, 0, s>>>(odd, nodd, classes, stride, nwords); break;
    case 210: {
      gather_kernel<210><<<(unsigned)blocks, kGatherThreads, 0, s>>>(odd, nodd, classes, stride, nwords);
      break;
    }
    default: return cudaErrorInvalidValue;
  }
  return cudaGetLastError();
}

cudaError_t launch_counts(const CountArgs& a, uint32_t* odd, uint64_t nodd, uint64_t start, uint64_t count,
                          cudaStream_t s) {
  const uint64_t small = (count + 255) / 256;
  const uint64_t tasks = (uint64_t)a.npairs * a.groups * a.splits;
  const uint64_t blocks = (tasks + kCountWarps - 1) / kCountWarps;
  if (blocks > 0x7fffffffull || small > 0x7fffffffull) return cudaErrorInvalidValue;
  counts_small_kernel<<<(unsigned)small, 256, 0, s>>>(odd, nodd, start, count, a.modulus, a.out);
  if (blocks) counts_kernel<<<(unsigned)blocks, kCountThreads, 0, s>>>(a);
  return cudaGetLastError();
}

}  // namespace gb
