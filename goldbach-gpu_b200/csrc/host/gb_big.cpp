// gb_big.cpp -- C-ABI entry point for even n beyond 2^64 (big_check).
//
// The reference's big_check (src/big_check.cpp:35-144) sieves the primes up
// to 1e7 on the host and runs GMP's mpz_probab_prime_p(n - p, 25) on OpenMP
// threads in batches of 1000 primes, keeping the first success.  Here the
// candidates come from the resident prime table in batches sized by n's length:
// the filter kernel drops q = n - p with a factor below kBigTrialBound (from
// n mod r, computed here once), the base-2 kernel tests the survivors, the
// bases kernel runs the other 11 bases on the smallest base-2 passer
// (kernels/big.cu), and the smallest passer no base rejects, in the first
// batch that has one, is the minimal p.
#include <algorithm>
#include <cstring>
#include <vector>

#include "gb_ctx.h"

namespace gb {

// Candidates per batch: two for each bit of n (one in 0.35 bits is prime, so
// about six of a batch are), 512 to kBigBatch.  A test of the batch beyond the
// first prime is of no use, and more than a warp per SM slows the others: 8192
// for every n against this, 512 bits 1.03 -> 0.82 ms, 1024 4.6 -> 3.5, 2048 20.0 ->
// 15.3; three a bit 0.83, 3.7 and 18.4.
constexpr uint32_t kBigBatch = 8192;
constexpr uint32_t kBatchPerBit = 2;
constexpr uint32_t kBigTrialBound = 4096;     // trial primes below this

gb_status big_impl(gb_ctx* c, Workspace& w, const uint32_t* n_limbs, uint32_t nlimbs,
                   uint64_t p_limit, uint64_t* p_out, uint32_t* q_limbs, gb_big_result* res) {
  if (!n_limbs || !p_out || nlimbs == 0) return fail(w, GB_EINVAL, "null argument");
  uint32_t m = nlimbs;
  while (m > 0 && n_limbs[m - 1] == 0) --m;
  if (m > GB_BIG_MAX_LIMBS) return fail(w, GB_EINVAL, "n has more than GB_BIG_MAX_LIMBS limbs");
  if (m == 0 || (n_limbs[0] & 1) || (m == 1 && n_limbs[0] < 4))
    return fail(w, GB_EINVAL, "n must be even and >= 4");
  if (!p_limit) p_limit = GB_PHASE2_LIMIT_DEFAULT;
  if (p_limit > 0xfffffffbull) return fail(w, GB_EINVAL, "p_limit above 2^32");
  gb_big_result r{};
  if (q_limbs) std::memset(q_limbs, 0, nlimbs * 4);
  if (m <= 2) {  // below 2^64: the deterministic single-n path
    const uint64_t n = m == 1 ? n_limbs[0] : ((uint64_t)n_limbs[1] << 32 | n_limbs[0]);
    uint64_t p = 0, q = 0;
    gb_single_opts so{};
    so.p_limit = p_limit;
    gb_single_result sr{};
    gb_status st = single_impl(c, w, nullptr, &n, 1, &p, &q, &so, &sr);
    if (st != GB_OK) return st;
    *p_out = p;
    if (q_limbs && p) {
      q_limbs[0] = (uint32_t)q;
      if (nlimbs > 1) q_limbs[1] = (uint32_t)(q >> 32);
    }
    r.candidates = 1;
    r.device_ms = sr.device_ms;
    if (res) *res = r;
    return GB_OK;
  }
  gb_status st = ensure_primes(c, w, std::max<uint64_t>(p_limit, kBigTrialBound));
  if (st != GB_OK) return st;
  uint64_t np = 0;
  if ((st = count_le(c, w, p_limit, &np)) != GB_OK) return st;
  // trial primes 3 .. kBigTrialBound and n mod each (from the top limb down)
  std::vector<uint32_t> trial, nmod;
  for (uint32_t p : c->h_primes) {
    if (p < 3) continue;
    if (p >= kBigTrialBound) break;
    uint64_t rem = 0;
    for (uint32_t i = m; i-- > 0;) rem = ((rem << 32) | n_limbs[i]) % p;
    trial.push_back(p);
    nmod.push_back((uint32_t)rem);
  }
  // one upload: n, the trial primes, n mod each
  std::vector<uint32_t> up(n_limbs, n_limbs + m);
  up.insert(up.end(), trial.begin(), trial.end());
  up.insert(up.end(), nmod.begin(), nmod.end());
  Temps tmp(c, nullptr);
  void *d_up, *d_surv, *d_pass, *d_small;
  if ((st = ws_buffer(c, w, tmp, 0, up.size() * 4, &d_up)) != GB_OK ||
      (st = ws_buffer(c, w, tmp, 1, kBigBatch / 8, &d_surv)) != GB_OK ||
      (st = ws_buffer(c, w, tmp, 2, kBigBatch * 4, &d_pass)) != GB_OK ||
      (st = ws_buffer(c, w, tmp, 3, 64, &d_small)) != GB_OK)
    return st;
  // the device's figures of a batch, in this order behind the tests' count
  struct Figures {
    unsigned long long tests;
    uint32_t npass, specfail, fail, minpass;
  };
  Figures* fig = (Figures*)d_small;
  BigArgs a{};
  a.n = (const uint32_t*)d_up;
  a.nl = m;
  uint32_t bits = 32 * m;
  while (!((n_limbs[m - 1] >> ((bits - 1) & 31)) & 1u)) --bits;
  a.limbs = (bits + 2 + 31) / 32;  // R >= 4n
  a.rl = big_r_lanes(a.limbs);
  a.primes = c->d_primes;
  a.p_lim = p_limit;
  a.trial = a.n + m;
  a.nmod = a.trial + trial.size();
  a.ntrial = (uint32_t)trial.size();
  a.surv = (uint32_t*)d_surv;
  a.pass = (uint32_t*)d_pass;
  a.npass = &fig->npass;
  a.minpass = &fig->minpass;
  a.specfail = &fig->specfail;
  a.fail = &fig->fail;
  a.mr_tests = &fig->tests;
  cudaStream_t s = c->stream;
  cudaError_t e = cudaSuccess;
  auto chk = [&](cudaError_t x) {
    if (e == cudaSuccess && x != cudaSuccess) e = x;
  };
  chk(cudaMemcpyAsync(d_up, up.data(), up.size() * 4, cudaMemcpyHostToDevice, s));
  chk(cudaMemsetAsync(d_small, 0, 64, s));
  chk(cudaEventRecord(w.ev0, s));
  Figures* h = (Figures*)w.h_stage;  // pinned
  *h = Figures{};  // (it holds an earlier call's figures, and np <= 1 reads none)
  uint32_t best = 0xffffffffu;
  uint64_t k0 = 1;  // p = 2 leaves q = n - 2 even
  uint32_t pk = 0;
  auto read = [&]() {
    chk(cudaMemcpyAsync(h, fig, sizeof(Figures), cudaMemcpyDeviceToHost, s));
    chk(cudaStreamSynchronize(s));
  };
  const uint32_t batch = std::min<uint32_t>(kBigBatch, std::max<uint32_t>(512, kBatchPerBit * bits));
  while (k0 < np && e == cudaSuccess) {
    const uint32_t kc = (uint32_t)std::min<uint64_t>(batch, np - k0);
    a.words = (kc + 31) / 32;
    chk(cudaMemsetAsync(&fig->npass, 0, 12, s));  // passers, specfail, fail
    chk(cudaMemsetAsync(&fig->minpass, 0xff, 4, s));
    chk(launch_big_filter(a, (uint32_t)k0, kc, s));
    chk(launch_big_base2(a, (uint32_t)k0, c->sm_count * 4, s));
    chk(launch_big_bases(a, (uint32_t)k0, 0xffffffffu, s));
    read();
    r.candidates += kc;
    if (e == cudaSuccess && h->npass) {
      best = h->minpass;
      if (h->fail) {  // a base rejected it: the other passers, in order
        std::vector<uint32_t> pass(h->npass);
        const uint32_t rejected = best;
        chk(cudaMemcpy(pass.data(), d_pass, pass.size() * 4, cudaMemcpyDeviceToHost));
        std::sort(pass.begin(), pass.end());
        best = 0xffffffffu;
        for (size_t j = 0; j < pass.size() && best == 0xffffffffu && e == cudaSuccess; ++j) {
          if (pass[j] == rejected) continue;
          chk(cudaMemsetAsync(&fig->fail, 0, 4, s));
          chk(launch_big_bases(a, (uint32_t)k0, pass[j], s));
          read();
          if (!h->fail) best = pass[j];
        }
      }
    }
    if (best != 0xffffffffu) {
      chk(cudaMemcpy(&pk, c->d_primes + k0 + best, 4, cudaMemcpyDeviceToHost));
      break;
    }
    k0 += kc;
  }
  chk(cudaEventRecord(w.ev1, s));
  const unsigned long long tests = e == cudaSuccess ? h->tests : 0;
  chk(cudaStreamSynchronize(s));
  if (e != cudaSuccess) return cuda_fail(w, e, "big n");
  float ms = 0;
  cudaEventElapsedTime(&ms, w.ev0, w.ev1);
  *p_out = best != 0xffffffffu ? pk : 0;
  if (q_limbs && *p_out) {  // q = n - p
    uint64_t borrow = *p_out;
    for (uint32_t i = 0; i < m; ++i) {
      const uint64_t v = (uint64_t)n_limbs[i] - (borrow & 0xffffffffu) - (borrow >> 32);
      q_limbs[i] = (uint32_t)v;
      borrow = ((v >> 32) & 1) << 32;
    }
  }
  r.mr_tests = tests;
  r.device_ms = ms;
  if (res) *res = r;
  return GB_OK;
}

}  // namespace gb
