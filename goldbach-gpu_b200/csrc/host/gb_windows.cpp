// gb_windows.cpp -- C-ABI entry point for batched windows.
//
// Many independent windows of consecutive even n (e.g. 4096 windows at
// offsets in [1e15, 1e18]) in one batch.  The reference has no batch mode:
// each window would be one `goldbach --start=A LIMIT` process with its own
// segment loop (src/goldbach.cu:420-485).  GB_WINDOWS_PERSISTENT runs the
// batch as one CUDA graph: the wide windows' class masks come from the
// large-prime pass, the narrower ones' from a short sieve and a primality test
// of every q it leaves (kernels/windows.cu); then range6_kernel in windows
// mode runs over every (window, chunk) item from one device work counter, and
// the device Phase 2 over what it leaves.  Windows of a few n, and small batches
// of narrow ones, go n by n through the single-n kernel instead.
// GB_WINDOWS_PLAIN runs the same launches window by window (the per-window
// launch pipeline, kept for comparison).
#include <algorithm>
#include <cmath>
#include <cstring>
#include <numeric>
#include <vector>

#include "gb_ctx.h"
#include "range_plan.h"

namespace gb {
// Primes up to this bound sieve each chunk's q-window in shared memory; the
// larger ones go through the large-prime pass (kernels/windows.cu), whose
// quotient estimate needs p > 2^20.  (2^22, 2^23 and 2^24 move marks from the
// pass to the chunks and cost there what they save here: 4096 windows 53.7 ms
// at 2^20, 56.4, 59.3 and 68 ms.)
constexpr uint64_t kWinChunkSieveBound = 1ull << 20;
// CTAs per SM of the large-prime pass (grid-stride over the primes: a fine
// grid evens out primes that visit many windows and primes that visit few)
constexpr uint64_t kLargeBlocksPerSM = 64;
// Halo of the windows' chunks: a minimal p beyond it goes to the device Phase 2.
// The largest minimal p known below 4e18 is 9781, and a 1024-n window's q-window is
// mostly halo (32768: 11 numbers of halo to one of the window).
constexpr uint32_t kWinHalo = 8192;
// Chunks of the windows are cut so that a small batch still fills the GPU,
// down to these widths; a tested window's chunks sieve no primes, so they can
// be narrower.
constexpr uint64_t kMinMaskedChunk = 1ull << 16;
constexpr double kMaskedFixed = 1e5;  // n that a masked range's chunk costs beside its own (balanced_chunk)
constexpr uint64_t kMinSievedChunk = 1ull << 15, kMinTestedChunk = 1ull << 13;

// The path of a window, by what it costs (results do not depend on it).
//   kTested: a short sieve and a primality test of every q left (about 16 ps
//     per n near 1e18, and some 100 ns for the halo);
//   kSieved: every sieving prime's first multiple (the large-prime pass: about
//     0.5 ps per prime, and 3 ps per n for its marks).
// So the line between the two lies at pi(sqrt(top)) / 30 n (4096 windows
// in [1e15, 1e18]: 53.7 ms at 20, 52.8 at 40, 61 at 80), pi(sqrt(top)) /
// mr_divisor where the caller sets it.  A third path takes a window n by n
// through the single-n kernel (per_n_windows).  mr_below = 1 sieves every window;
// another mr_below sends narrower windows n by n and sieves the others.
enum WinPath { kTested, kSieved };  // (ranges: range_masked below)
constexpr double kTestDivisor = 30.0;

static WinPath window_path(const gb_window& w, const gb_windows_opts& o) {
  if (o.mr_below) return kSieved;
  const uint64_t last = w.start + 2 * (w.count - 1);
  const double r = std::sqrt((double)last);
  if (r <= (double)kWinChunkSieveBound) return kSieved;  // no prime needs the large-prime pass
  const double div = o.mr_divisor ? (double)o.mr_divisor : kTestDivisor;
  const double lim = 1.1 * r / std::log(r) / div;  // pi(r) < 1.1 r / ln r here
  return (double)w.count >= lim ? kSieved : kTested;
}

// The windows that go n by n, which costs 60 us for the batch and 0.75 to 1.2 ns
// per n.  The other two paths cost 85 us (sieved, near 1e9) to 140 (tested) for
// the batch, and 0.13 to 0.31 us per window whatever its width.  Measured, n by n
// against the others, in us: 4096 windows of 100 n 301 / 681 near 1e9, 360 / 1256
// near 1e12, 474 / 1411 near 1e18, of 256 n 520 / 715, 634 / 1318, 880 / 1487; one
// window of 1 n near 1e12 65 / 116, of 1000 n near 1e18 72 / 151, of 16000 n 142 /
// 177, of 30000 193 / 178; 8 windows of 4000 n near 1e18 130 / 176, of 16000 255 /
// 178; 64 of 1000 n 158 / 181, of 2000 218 / 183.  So:
//   * a batch goes n by n as a whole when its windows have fewer than kPerNMax n,
//     or, where they would be tested, up to kPerNWide, and together not more than
//     kPerNBatch beside kPerNMax for each;
//   * in another batch the windows of fewer than kPerNMax n do when what they
//     save (half as much where they would be sieved) is worth kPerNBatch n, the
//     other path's fixed cost.
// n below 2^21 take the single-n kernel's plain path, a warp each (4096 windows of
// 100 n near 1e6 10.3 ms / 0.6): such windows are not taken.
// With an arena only windows of fewer than kPerNMax n do, for the memory that
// windows_request_bytes states.  few, and where this takes more than kPerNMost n
// (24 bytes each): tested windows of fewer than kPerNFew n alone.
constexpr uint64_t kPerNMax = 256, kPerNWide = 1ull << 14, kPerNBatch = 1ull << 16, kPerNMost = 1ull << 24;
constexpr uint64_t kPerNFew = 64;
constexpr uint64_t kPerNLeast = 1ull << 21;

static bool is_narrow(const gb_window& w) { return w.count < kPerNMax && w.start >= kPerNLeast; }

static std::vector<char> per_n_windows(const gb_window* w, size_t count, const gb_windows_opts& o, bool arena,
                                       bool few) {
  std::vector<char> per_n(count, 0);
  if (o.mr_below) {
    for (size_t i = 0; i < count; ++i) per_n[i] = w[i].count < o.mr_below && o.mr_below != 1;
    return per_n;
  }
  bool all = true;
  uint64_t total = 0, narrow = 0, saved = 0;  // n: of the batch, of the narrow windows, worth of going n by n
  for (size_t i = 0; i < count; ++i) {
    const uint64_t n = w[i].count;
    const bool tested = window_path(w[i], o) == kTested;
    per_n[i] = tested && n < kPerNFew;
    if (!is_narrow(w[i]) && (arena || !tested || n > kPerNWide)) all = false;
    total += std::min(n, kPerNWide);
    if (is_narrow(w[i])) {
      narrow += n;
      saved += (kPerNMax - n) >> (tested ? 0 : 1);
    }
  }
  all = all && total <= kPerNBatch + kPerNMax * count;
  if (few || (all ? total : narrow) > kPerNMost) return per_n;
  for (size_t i = 0; i < count; ++i) per_n[i] = all || (saved >= kPerNBatch && is_narrow(w[i]));
  return per_n;
}

// What the pipeline's options do not allow (null: nothing).
static const char* opts_error(const gb_windows_opts& o) {
  const uint32_t H = o.halo ? o.halo : kWinHalo, NE = o.chunk_evens ? o.chunk_evens : (1u << 20);
  if (H < 128 || H > (1u << 17) || (H & 63)) return "halo must be a multiple of 64 in [128, 2^17]";
  if (NE < 8192 || NE > (1u << 20) || (NE & (NE - 1))) return "chunk_evens must be a power of two in [2^13, 2^20]";
  if (o.block_threads && o.block_threads != 256 && o.block_threads != 512 && o.block_threads != 1024)
    return "block_threads must be 256, 512 or 1024";
  if (o.phase2_limit > GB_P_SMALL_MAX) return "phase2_limit must be <= 4e9";
  if (o.gpu_share_pct > 100) return "gpu_share_pct must be <= 100";
  return nullptr;
}

// The largest power of two up to `most` that cuts `total` n into at least
// `pieces` chunks, but at least `least`.
static uint32_t chunk_for(uint64_t total, uint64_t pieces, uint64_t least, uint64_t most) {
  uint64_t ne = most;
  while (ne > least && total / ne < pieces) ne >>= 1;
  return (uint32_t)ne;
}

// floor((A - H - 1) / 6) for A possibly below H (range.cu window_g0)
static int64_t host_window_g0(uint64_t A, uint32_t H) {
  if (A >= (uint64_t)H + 1) return (int64_t)((A - H - 1) / 6);
  return -(int64_t)(((uint64_t)H + 1 - A + 5) / 6);
}

// ---------------------------------------------------------------------------
// A range through the windows' kernels (range_impl): its segments, cut into
// pieces, are the windows of range6_kernel's work items, and runs of adjacent
// pieces share one mask, so the large-prime pass meets each prime once per run
// instead of once per chunk.  Runs and batches hold at most kRangeMaskEvens n,
// whose masks stay in L2.

// Largest prime the chunks sieve themselves: about the chunk's own width (a
// prime above a third of it marks a class less than once), and enough for the
// pass's quotient estimate of the primes beyond it.
static uint64_t masked_bound(uint64_t top, uint32_t ne) {
  return std::min<uint64_t>(kWinChunkSieveBound, std::max<uint64_t>({1ull << 14, (uint64_t)ne, (top / 6) >> 42}));
}

gb_status range_masked(gb_ctx* c, Workspace& ws, Temps& tmp, int slot, const std::vector<RangePiece>& segs,
                       RangeArgs a, uint32_t ne, uint64_t root, cudaStream_t s, int* launches) {
  const uint32_t H = a.s.halo;
  // pieces and the runs of adjacent ones
  struct Run {
    size_t p0, p1;  // pieces
    WinDesc6 mask;
  };
  std::vector<WinDesc6> desc;
  std::vector<Run> runs;
  uint64_t run_n = 0, total = 0, top = 0;
  for (const RangePiece& g : segs)
    for (uint64_t j = 0; j < g.count; j += kRangeMaskEvens) {
      WinDesc6 d{};
      d.start = g.start + 2 * j;
      d.count = std::min(kRangeMaskEvens, g.count - j);
      d.out_off = g.out_off + j;
      d.q_top = d.start + 2 * (d.count - 1);
      d.orig = g.unit;
      const bool joins = !desc.empty() && desc.back().q_top + 2 == d.start && run_n + d.count <= kRangeMaskEvens;
      if (!joins) {
        runs.push_back(Run{desc.size(), desc.size(), WinDesc6{}});
        run_n = 0;
      }
      run_n += d.count;
      total += d.count;
      top = std::max(top, d.q_top);
      desc.push_back(d);
      runs.back().p1 = desc.size();
    }
  if (!ne) {
    // one batch's pieces: its segments, or its share of a longer one
    const uint64_t n = std::min(total, kRangeMaskEvens);
    const uint64_t len = std::min<uint64_t>(segs[0].count, kRangeMaskEvens);
    ne = balanced_chunk(n / len, len, n % len, kMaskedFixed, c->sm_count, kMinMaskedChunk, a.chunk_evens);
  }
  a.chunk_evens = ne;
  a.nbw = range6_words(H, ne);
  const uint64_t bound = masked_bound(top, ne);
  uint64_t nsmall = 0, kc = 0;
  const uint64_t nlarge = count_bound(c, root);  // (the pass stops at each window's top)
  gb_status st;
  if ((st = count_le(c, ws, std::min(bound, root), &nsmall)) != GB_OK ||
      (st = count_le(c, ws, (H / 6 + ne / 3) / 32, &kc)) != GB_OK)
    return st;
  nsmall = std::max<uint64_t>(nsmall, kWheelPrimeCount + 1);
  a.kcoop = (uint32_t)std::max<uint64_t>(std::min(kc, nsmall), kWheelPrimeCount + 1);
  // masks, batch by batch in the same buffer
  struct Batch {
    size_t r0, r1;
    uint64_t words, items, off0;  // off0: first entry of its chunk offsets
  };
  std::vector<Batch> batches;
  std::vector<WinDesc6> masks;
  std::vector<WinLarge> wl;
  std::vector<uint64_t> coff;
  uint64_t batch_n = 0, max_words = 0;
  for (size_t r = 0; r < runs.size(); ++r) {
    Run& u = runs[r];
    uint64_t n = 0;
    for (size_t p = u.p0; p < u.p1; ++p) n += desc[p].count;
    if (batches.empty() || batch_n + n > kRangeMaskEvens) {
      batches.push_back(Batch{r, r, 0, 0, coff.size()});
      coff.push_back(0);
      batch_n = 0;
    }
    Batch& b = batches.back();
    batch_n += n;
    b.r1 = r + 1;
    const int64_t g0 = host_window_g0(desc[u.p0].start, H);
    uint64_t lw = 0;
    for (size_t p = u.p0; p < u.p1; ++p) {
      WinDesc6& d = desc[p];
      d.g0 = g0;
      d.lbase = b.words;
      d.ne = ne;
      d.nsieve = (uint32_t)nsmall;
      const uint64_t chunks = (d.count + ne - 1) / ne;
      // the mask words the last two chunks read, from the mask's base on (as in
      // windows_sieve_impl)
      for (uint64_t ci = chunks >= 2 ? chunks - 2 : 0; ci < chunks; ++ci) {
        const uint64_t cnt = std::min<uint64_t>(ne, d.count - ci * ne);
        const uint64_t nwords = std::min<uint64_t>(a.nbw, (H / 6 + cnt / 3 + 96 + 31) / 32 + 2);
        const int64_t gc = host_window_g0(d.start + 2 * (uint64_t)ne * ci, H);
        lw = std::max(lw, ((uint64_t)(gc - g0) >> 5) + nwords + 2);
      }
      b.items += chunks;
      coff.push_back(b.items);
    }
    u.mask = desc[u.p0];
    u.mask.lwords = (uint32_t)((lw + 3) & ~3ull);
    u.mask.q_top = desc[u.p1 - 1].q_top;
    for (size_t p = u.p0; p < u.p1; ++p) desc[p].lwords = u.mask.lwords;
    b.words += 2ull * u.mask.lwords;
    max_words = std::max(max_words, b.words);
    masks.push_back(u.mask);
    wl.push_back(WinLarge{(double)g0, 0u - (uint32_t)(uint64_t)g0, u.mask.lwords * 32});
  }
  // one upload: descriptors, masks, records, chunk offsets
  const size_t o_mask = desc.size() * sizeof(WinDesc6), o_wl = (o_mask + masks.size() * sizeof(WinDesc6) + 15) & ~size_t(15);
  const size_t o_off = o_wl + wl.size() * sizeof(WinLarge), bytes = o_off + coff.size() * 8;
  std::vector<char> up_big(bytes <= kIoBytes ? 0 : bytes);  // pageable: staged at the copy
  char* const up = up_big.empty() ? ws.h_io : up_big.data();
  std::memcpy(up, desc.data(), desc.size() * sizeof(WinDesc6));
  std::memcpy(up + o_mask, masks.data(), masks.size() * sizeof(WinDesc6));
  std::memcpy(up + o_wl, wl.data(), wl.size() * sizeof(WinLarge));
  std::memcpy(up + o_off, coff.data(), coff.size() * 8);
  void *d_up, *d_mask;
  if ((st = ws_buffer(c, ws, tmp, slot, bytes, &d_up)) != GB_OK ||
      (st = ws_buffer(c, ws, tmp, slot + 1, max_words * 4, &d_mask)) != GB_OK)
    return st;
  int bps = range_max_blocks_per_sm(a);
  if (bps < 1) bps = 1;
  const uint64_t grid_max = (uint64_t)c->sm_count * bps;
  a.surv_cap = a.nbw;
  void* scratch = nullptr;
  if ((st = ws_scratch(c, ws, (size_t)grid_max * 6 * a.surv_cap * sizeof(uint2), &scratch)) != GB_OK) return st;
  a.surv = (uint2*)scratch;
  a.lmask = (const uint32_t*)d_mask;
  WinLargeArgs la{};
  la.primes = c->d_primes;
  la.magic = c->d_magic;
  la.a15 = c->d_a15;
  la.k0 = (uint32_t)nsmall;
  la.k1 = (uint32_t)std::max<uint64_t>(nlarge, nsmall);
  la.lmask = (uint32_t*)d_mask;
  la.pairs = a.s.ctr + kCtrPairs;
  const uint64_t np = la.k1 - la.k0;
  const int gl = (int)std::max<uint64_t>(1, std::min<uint64_t>((np + 511) / 512, (uint64_t)c->sm_count * kLargeBlocksPerSM));
  cudaError_t e = cudaMemcpyAsync(d_up, up, bytes, cudaMemcpyHostToDevice, s);
  auto chk = [&](cudaError_t x) {
    if (e == cudaSuccess && x != cudaSuccess) e = x;
  };
  const WinDesc6* dd = (const WinDesc6*)d_up;
  for (const Batch& b : batches) {
    chk(cudaMemsetAsync(d_mask, 0xff, b.words * 4, s));
    if (&b != &batches[0]) chk(cudaMemsetAsync(a.s.ctr + kCtrWork, 0, 8, s));
    la.win = (const WinDesc6*)((char*)d_up + o_mask) + b.r0;
    la.wl = (const WinLarge*)((char*)d_up + o_wl) + b.r0;
    la.w_lo = 0;
    la.w_hi = (uint32_t)(b.r1 - b.r0);
    if (np) chk(launch_win_large(la, gl, s));
    a.win = dd + runs[b.r0].p0;
    a.nwin = (uint32_t)(runs[b.r1 - 1].p1 - runs[b.r0].p0);
    a.chunk_off = (const uint64_t*)((char*)d_up + o_off) + b.off0;
    a.total_items = b.items;
    chk(launch_range(a, (int)std::min(grid_max, b.items), s));
    *launches += np ? 2 : 1;
  }
  return e == cudaSuccess ? GB_OK : cuda_fail(ws, e, "range (masked)");
}

// The sieve pipeline over windows w[0..count).
static gb_status windows_sieve_impl(gb_ctx* c, Workspace& ws, Arena* arena, const gb_window* w,
                                    size_t count, const gb_windows_opts* opts, gb_window_result* res,
                                    uint32_t* min_p_concat, gb_windows_summary* sum) {
  if (count && !w) return fail(ws, GB_EINVAL, "null windows");
  gb_windows_opts o{};
  if (opts) o = *opts;
  if (o.mode != GB_WINDOWS_PERSISTENT && o.mode != GB_WINDOWS_PLAIN)
    return fail(ws, GB_EINVAL, "unknown windows mode");
  if (o.on_device) return fail(ws, GB_EINVAL, "windows: on_device outputs are not supported");
  if (sum) std::memset(sum, 0, sizeof *sum);
  if (count == 0) return GB_OK;
  if (count > 0xffffffffull) return fail(ws, GB_EINVAL, "too many windows");
  const uint32_t H = o.halo ? o.halo : kWinHalo;
  uint32_t NE = o.chunk_evens ? o.chunk_evens : (1u << 20);
  if (const char* bad = opts_error(o)) return fail(ws, GB_EINVAL, bad);
  if (min_p_concat && NE > kMinpChunk) NE = kMinpChunk;  // per-n output: smaller chunks
  const uint64_t p_lim = o.phase2_limit ? o.phase2_limit : GB_PHASE2_LIMIT_DEFAULT;
  const uint64_t large_per_sm = o.large_ctas_per_sm ? o.large_ctas_per_sm : kLargeBlocksPerSM;
  const uint64_t share = o.gpu_share_pct ? o.gpu_share_pct : 100;
  std::vector<uint32_t> order(count);
  std::vector<char> tested(count);
  uint64_t total_n = 0, n_tested = 0, q_max = 0, q_sieved = 0;
  for (size_t i = 0; i < count; ++i) {
    if (w[i].start < 4 || (w[i].start & 1) || w[i].count == 0)
      return fail(ws, GB_EINVAL, "window start must be even and >= 4, count >= 1");
    const uint64_t last = w[i].start + 2 * (w[i].count - 1);
    if (w[i].count > GB_WINDOW_MAX_COUNT) return fail(ws, GB_EINVAL, "window wider than GB_WINDOW_MAX_COUNT");
    if (last < w[i].start) return fail(ws, GB_EINVAL, "window passes 2^64");
    tested[i] = window_path(w[i], o) == kTested;
    if (tested[i]) n_tested += w[i].count;
    else q_sieved = std::max(q_sieved, last);
    q_max = std::max(q_max, last);
    total_n += w[i].count;
  }
  // a sieved window needs every prime up to its top's root, a tested one only
  // those of its presieve (below kHostPrimeLimit, which every table covers)
  const uint64_t root = isqrt_u64(q_max), root_sieved = isqrt_u64(q_sieved);
  gb_status st = ensure_primes(c, ws, std::max<uint64_t>({p_lim, (uint64_t)H, root_sieved + 2, kWinChunkSieveBound}));
  if (st != GB_OK) return st;
  // descriptors: the sieved windows first, sorted by top q so that a prime
  // visits a suffix of them, then the tested ones
  std::iota(order.begin(), order.end(), 0u);
  std::sort(order.begin(), order.end(), [&](uint32_t x, uint32_t y) {
    if (tested[x] != tested[y]) return tested[x] < tested[y];
    return w[x].start + 2 * (w[x].count - 1) < w[y].start + 2 * (w[y].count - 1);
  });
  const size_t nsw = count - std::count(tested.begin(), tested.end(), 1);  // sieved windows
  // chunk widths of the two kinds
  const uint64_t slots = 4ull * c->sm_count;
  uint32_t ne_s = NE, ne_t = NE;
  if (!o.chunk_evens) {
    ne_s = chunk_for(total_n - n_tested, slots, std::min<uint64_t>(kMinSievedChunk, NE), NE);
    ne_t = chunk_for(n_tested, slots, std::min<uint64_t>(kMinTestedChunk, NE), std::min<uint64_t>(1u << 17, NE));
    NE = nsw == 0 ? ne_t : nsw == count ? ne_s : std::max(ne_s, ne_t);
  }
  const uint32_t nbw = range6_words(H, NE);
  std::vector<uint64_t> out_off(count + 1, 0);
  for (size_t i = 0; i < count; ++i) out_off[i + 1] = out_off[i] + w[i].count;
  std::vector<WinDesc6> desc(count);
  std::vector<WinLarge> wl(count);
  std::vector<uint64_t> chunk_off(count + 1, 0), chunk_one(2 * count, 0);
  std::vector<uint64_t> test_one(4 * (count - nsw), 0);  // plain mode: each tested window's own offsets
  std::vector<uint64_t> tile_off(count - nsw + 1, 0), run_off(count - nsw + 1, 0);
  uint64_t nsmall = 0;
  if ((st = count_le(c, ws, std::min<uint64_t>(kWinChunkSieveBound, root), &nsmall)) != GB_OK) return st;
  nsmall = std::max<uint64_t>(nsmall, kWheelPrimeCount + 1);
  uint64_t lwords_total = 0, lwords_sieved = 0;
  for (size_t r = 0; r < count; ++r) {
    const uint32_t i = order[r];
    WinDesc6& d = desc[r];
    d.start = w[i].start;
    d.count = w[i].count;
    d.out_off = out_off[i];
    d.q_top = d.start + 2 * (d.count - 1);
    d.g0 = host_window_g0(d.start, H);
    d.orig = i;
    d.ne = r < nsw ? ne_s : ne_t;
    d.nsieve = r < nsw ? (uint32_t)nsmall : 0;
    const uint64_t chunks = (d.count + d.ne - 1) / d.ne;
    // a chunk reads nwords + 1 mask words from its own base on (nwords as in
    // range6_kernel: the words its search can read for a real n); the mask
    // ends there, so the large-prime pass marks no bit nobody reads
    auto reach = [&](uint64_t ci) {  // mask words chunk ci reads, from the window base
      const uint64_t cnt = std::min<uint64_t>(d.ne, d.count - ci * d.ne);
      const uint64_t nbits = H / 6 + cnt / 3 + 96;
      const uint64_t nwords = std::min<uint64_t>(nbw, (nbits + 31) / 32 + 2);
      const int64_t gc = host_window_g0(d.start + 2 * (uint64_t)d.ne * ci, H);
      return ((uint64_t)(gc - d.g0) >> 5) + nwords + 2;
    };
    // the last full chunk or the (possibly short) last one reaches furthest
    uint64_t lw = reach(chunks - 1);
    if (chunks >= 2) lw = std::max(lw, reach(chunks - 2));
    d.lwords = (uint32_t)((lw + 3) & ~3ull);
    d.lbase = lwords_total;
    lwords_total += 2ull * d.lwords;
    if (r < nsw) lwords_sieved = lwords_total;
    wl[r].gd = (double)d.g0;
    wl[r].ngl = 0u - (uint32_t)(uint64_t)d.g0;
    wl[r].lbits = d.g0 >= (int64_t)(1ll << 30) && d.lwords < (1u << 27) / 32 ? d.lwords * 32 : kLargeExact;
    chunk_off[r + 1] = chunk_off[r] + chunks;
    chunk_one[2 * r + 1] = chunks;
  }
  // presieve tiles and test runs of the tested windows
  WinTestArgs ta{};
  uint64_t tile_words = kTileWordsMax;
  while (tile_words > 64 && (lwords_total - lwords_sieved) / 2 / tile_words < slots) tile_words >>= 1;
  ta.tile_words = (uint32_t)tile_words;
  for (size_t r = nsw; r < count; ++r) {
    const uint64_t lw = desc[r].lwords;
    tile_off[r - nsw + 1] = tile_off[r - nsw] + (lw + tile_words - 1) / tile_words;
    run_off[r - nsw + 1] = run_off[r - nsw] + 2 * ((lw + 31) / 32);
    test_one[4 * (r - nsw) + 1] = tile_off[r - nsw + 1] - tile_off[r - nsw];
    test_one[4 * (r - nsw) + 3] = run_off[r - nsw + 1] - run_off[r - nsw];
  }
  for (int k = 0; k < kTileLogs; ++k) {
    // a prime costs a tile about 12 instructions, a q left of the tile's 192
    // numbers a word about 2400 for its base-2 test: the derivatives meet near
    // ten primes' reach per number
    const uint64_t bound = std::min<uint64_t>({root, 1920ull << k, kHostPrimeLimit / 2});
    uint64_t n = 0;
    if ((st = count_le(c, ws, bound, &n)) != GB_OK) return st;
    ta.nsieve[k] = (uint32_t)std::max<uint64_t>(n, kWheelPrimeCount + 1);
  }
  uint64_t ns = 0, kc = 0, kct = 0;
  const uint64_t kf = count_bound(c, p_lim), nlarge = count_bound(c, root_sieved);
  if ((st = count_le(c, ws, std::min<uint64_t>(H - 13, p_lim), &ns)) != GB_OK ||
      (st = count_le(c, ws, (H / 6 + NE / 3) / 64, &kc)) != GB_OK ||
      (st = count_le(c, ws, tile_words / 2, &kct)) != GB_OK)
    return st;

  // one upload: descriptors, records, chunk offsets, the tested windows' tile
  // and run offsets, and the plain mode's offsets of single windows
  const bool plain = o.mode == GB_WINDOWS_PLAIN;
  const size_t o_wl = (count * sizeof(WinDesc6) + 15) & ~size_t(15);
  const size_t o_coff = o_wl + count * sizeof(WinLarge);
  const size_t o_tile = o_coff + (count + 1) * 8, o_run = o_tile + tile_off.size() * 8;
  const size_t o_cone = o_run + run_off.size() * 8, o_tone = o_cone + (plain ? 2 * count * 8 : 0);
  const size_t up_bytes = o_tone + (plain ? test_one.size() * 8 : 0);
  ws.buf_used = 0;  // (the other path's part of the batch is complete, and so is an earlier batch)
  // results: sum and largest minimal p and failures of each window
  const size_t res_bytes = count * 20;
  Temps tmp(c, arena);
  void *d_up, *d_lmask, *d_res, *d_minp = nullptr;
  if ((st = ws_buffer(c, ws, tmp, 0, up_bytes, &d_up)) != GB_OK ||
      (st = ws_buffer(c, ws, tmp, 1, res_bytes, &d_res)) != GB_OK ||
      (st = ws_buffer(c, ws, tmp, 2, lwords_total * 4, &d_lmask)) != GB_OK ||
      (min_p_concat && (st = ws_buffer(c, ws, tmp, 3, total_n * 4, &d_minp)) != GB_OK))
    return st;
  std::vector<char> up_big(up_bytes <= kIoBytes ? 0 : up_bytes);  // pageable: staged at the copy
  char* const up = up_big.empty() ? ws.h_io : up_big.data();
  std::memcpy(up, desc.data(), count * sizeof(WinDesc6));
  std::memcpy(up + o_wl, wl.data(), count * sizeof(WinLarge));
  std::memcpy(up + o_coff, chunk_off.data(), (count + 1) * 8);
  std::memcpy(up + o_tile, tile_off.data(), tile_off.size() * 8);
  std::memcpy(up + o_run, run_off.data(), run_off.size() * 8);
  if (plain) {
    std::memcpy(up + o_cone, chunk_one.data(), 2 * count * 8);
    if (!test_one.empty()) std::memcpy(up + o_tone, test_one.data(), test_one.size() * 8);
  }
  const void* d_desc = d_up;
  const void* d_wl = (char*)d_up + o_wl;
  const uint64_t* d_coff = (const uint64_t*)((char*)d_up + o_coff);
  const uint64_t* d_cone = (const uint64_t*)((char*)d_up + o_cone);
  const uint64_t* d_tone = (const uint64_t*)((char*)d_up + o_tone);
  void* const d_psum = d_res;
  void* const d_maxp = (char*)d_res + count * 8;
  void* const d_fail = (char*)d_res + count * 16;

  RangeArgs a{};
  SearchParams& sp = a.s;
  sp.halo = H;
  sp.nsearch = (uint32_t)ns;
  sp.kfb = (uint32_t)std::min<uint64_t>(kf, 0xffffffffu);
  sp.p_lim = p_lim;
  sp.p_small = p_lim;
  sp.primes = c->d_primes;
  sp.nprimes = c->nprimes;
  sp.ctr = ws.ctr;
  sp.unit_failures = (uint32_t*)d_fail;
  sp.unit_maxp = (unsigned long long*)d_maxp;
  sp.unit_psum = (unsigned long long*)d_psum;
  sp.minp = (uint32_t*)d_minp;
  sp.queue = ws.queue;
  sp.queue_cap = ws.queue_cap;
  a.chunk_evens = NE;
  a.threads = o.block_threads;
  a.nbw = nbw;
  a.magic = c->d_magic;
  a.nsieve = (uint32_t)nsmall;
  a.kcoop = (uint32_t)std::max<uint64_t>(std::min(kc, nsmall), kWheelPrimeCount + 1);
  a.wheel6 = c->d_wheel6;
  a.a15 = c->d_a15;
  a.win = (const WinDesc6*)d_desc;
  a.chunk_off = d_coff;
  a.nwin = (uint32_t)count;
  a.lmask = (const uint32_t*)d_lmask;
  a.total_items = chunk_off[count];
  WinLargeArgs la{};
  la.win = (const WinDesc6*)d_desc;
  la.wl = (const WinLarge*)d_wl;
  la.w_lo = 0;
  la.w_hi = (uint32_t)nsw;
  la.primes = c->d_primes;
  la.magic = c->d_magic;
  la.a15 = c->d_a15;
  la.k0 = (uint32_t)nsmall;
  la.k1 = (uint32_t)std::max<uint64_t>(nlarge, la.k0);
  la.lmask = (uint32_t*)d_lmask;
  la.pairs = sp.ctr + kCtrPairs;
  const size_t ntw = count - nsw;  // tested windows
  ta.win = (const WinDesc6*)d_desc + nsw;
  ta.tile_off = (const uint64_t*)((char*)d_up + o_tile);
  ta.run_off = (const uint64_t*)((char*)d_up + o_run);
  ta.nwin = (uint32_t)ntw;
  ta.tiles = tile_off[ntw];
  ta.runs = run_off[ntw];
  ta.kcoop = (uint32_t)std::max<uint64_t>(kct, kWheelPrimeCount + 1);
  ta.primes = c->d_primes;
  ta.magic = c->d_magic;
  ta.a15 = c->d_a15;
  ta.wheel6 = c->d_wheel6;
  ta.lmask = (uint32_t*)d_lmask;
  ta.ctr = sp.ctr + kCtrTest;

  const int sm = c->sm_count;
  int bps = range_max_blocks_per_sm(a);
  if (bps < 1) bps = 1;
  // CTAs the chunk kernel may keep resident: its share of the GPU
  const uint64_t grid_max = std::max<uint64_t>(1, (uint64_t)sm * bps * share / 100);
  a.surv_cap = nbw;
  {
    void* p = nullptr;
    if ((st = ws_scratch(c, ws, (size_t)grid_max * 6 * a.surv_cap * sizeof(uint2), &p)) != GB_OK) return st;
    a.surv = (uint2*)p;
  }
  const uint64_t np = la.k1 - la.k0;
  // the large-prime pass is not capped by the share: its CTAs are short
  // (a few primes each, grid-stride) and free their slots as they finish,
  // where higher-priority work takes them; a capped grid left it with too
  // few warps per SM to hide its loads
  const int g_pre = (int)std::max<uint64_t>(1, std::min<uint64_t>(ta.tiles, (uint64_t)sm * kPresieveCtasPerSm * share / 100));
  const int g_test = (int)std::max<uint64_t>(1, std::min<uint64_t>((ta.runs + 7) / 8, (uint64_t)sm * kWinTestCtasPerSm * share / 100));
  const int gl = (int)std::max<uint64_t>(1, std::min<uint64_t>((np + 255) / 256, (uint64_t)sm * large_per_sm));

  cudaStream_t s = o.stream ? (cudaStream_t)o.stream : c->stream;
  cudaError_t e = cudaSuccess;
  auto chk = [&](cudaError_t x) {
    if (e == cudaSuccess && x != cudaSuccess) e = x;
  };
  chk(cudaMemcpyAsync(d_up, up, up_bytes, cudaMemcpyHostToDevice, s));
  chk(cudaMemsetAsync(d_res, 0, res_bytes, s));
  chk(cudaMemsetAsync(sp.ctr, 0, kCtrCount * 8, s));
  chk(cudaMemsetAsync(sp.ctr + kCtrFirstFail, 0xff, 8, s));
  int launches = 0;
  float large_ms = 0, search_ms = 0;
  chk(cudaEventRecord(ws.ev0, s));
  if (o.mode == GB_WINDOWS_PERSISTENT) {
    // The batch's launches as one CUDA graph: captured per call (the
    // arguments change), applied to the workspace's executable graph by an
    // in-place update -- the topology repeats from batch to batch, so the
    // graph is instantiated once and relaunched -- and launched as one unit.
    // A caller that is itself capturing the stream gets the launches inline.
    cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;
    chk(cudaStreamIsCapturing(s, &cs));
    const bool graph = e == cudaSuccess && cs == cudaStreamCaptureStatusNone;
    auto mark = [&](cudaEvent_t ev) {  // timing events: nodes of the graph
      chk(graph ? cudaEventRecordWithFlags(ev, s, cudaEventRecordExternal) : cudaEventRecord(ev, s));
    };
    if (graph) chk(cudaStreamBeginCapture(s, cudaStreamCaptureModeThreadLocal));
    // every kernel is there in every batch, with a grid of one where it has no
    // work: another topology would have the graph instantiated anew, as another
    // number of mask groups does (each of them takes longer than that)
    chk(cudaMemsetAsync(d_lmask, 0xff, std::max<uint64_t>(lwords_sieved, 1) * 4, s));
    mark(ws.ek0);
    size_t r = 0;
    do {  // groups of windows whose masks stay in L2 together
      WinLargeArgs l = la;
      l.w_lo = (uint32_t)r;
      for (uint64_t bytes = 0; r < nsw && (r == l.w_lo || bytes + 8ull * desc[r].lwords <= kLargeGroupBytes); ++r)
        bytes += 8ull * desc[r].lwords;
      l.w_hi = (uint32_t)r;
      if (!nsw) l.k1 = l.k0;
      chk(launch_win_large(l, nsw ? gl : 1, s));
      ++launches;
    } while (r < nsw);
    mark(ws.ek1);
    chk(launch_win_presieve(ta, g_pre, s));
    chk(launch_win_test(ta, g_test, s));
    launches += 2;
    const int grid = (int)std::max<uint64_t>(1, std::min<uint64_t>(grid_max, a.total_items));
    chk(launch_range(a, grid, s));
    mark(ws.ek2);
    chk(launch_fallback(sp, sm * 4, s));
    launches += 2;
    if (graph) {
      cudaGraph_t g = nullptr;
      const cudaError_t ec = cudaStreamEndCapture(s, &g);  // ends the capture in every case
      chk(ec);
      if (e == cudaSuccess) {
        cudaGraphExecUpdateResultInfo info{};
        if (!ws.win_exec || cudaGraphExecUpdate(ws.win_exec, g, &info) != cudaSuccess) {
          cudaGetLastError();  // another topology: instantiate anew
          if (ws.win_exec) cudaGraphExecDestroy(ws.win_exec);
          ws.win_exec = nullptr;
          chk(cudaGraphInstantiate(&ws.win_exec, g, 0));
        }
        if (e == cudaSuccess) chk(cudaGraphLaunch(ws.win_exec, s));
      }
      if (g) cudaGraphDestroy(g);
    }
  } else {
    for (uint32_t r = 0; r < count && e == cudaSuccess; ++r) {
      const WinDesc6& d = desc[r];
      chk(cudaMemsetAsync(sp.ctr + kCtrWork, 0, 8, s));
      chk(cudaMemsetAsync(sp.ctr + kCtrQueue, 0, 8, s));
      if (r < nsw) {
        chk(cudaMemsetAsync((uint32_t*)d_lmask + d.lbase, 0xff, 2ull * d.lwords * 4, s));
        WinLargeArgs l1 = la;
        l1.w_lo = r;
        l1.w_hi = r + 1;
        if (l1.k1 > l1.k0 && d.q_top >= kWinChunkSieveBound * kWinChunkSieveBound) {
          chk(launch_win_large(l1, gl, s));
          ++launches;
        }
      } else {
        WinTestArgs t1 = ta;  // one window, with offsets of its own
        t1.win = ta.win + (r - nsw);
        t1.nwin = 1;
        t1.tiles = tile_off[r - nsw + 1] - tile_off[r - nsw];
        t1.runs = run_off[r - nsw + 1] - run_off[r - nsw];
        t1.tile_off = d_tone + 4 * (r - nsw);
        t1.run_off = t1.tile_off + 2;
        chk(cudaMemsetAsync(ta.ctr, 0, 8, s));
        chk(launch_win_presieve(t1, (int)std::min<uint64_t>(t1.tiles, g_pre), s));
        chk(launch_win_test(t1, (int)std::min<uint64_t>((t1.runs + 7) / 8, g_test), s));
        launches += 2;
      }
      RangeArgs a1 = a;
      a1.win = (const WinDesc6*)d_desc + r;
      a1.chunk_off = d_cone + 2 * r;
      a1.nwin = 1;
      a1.total_items = chunk_one[2 * r + 1];
      chk(launch_range(a1, (int)std::min<uint64_t>(grid_max, a1.total_items), s));
      chk(launch_fallback(sp, std::max(1, sm / 4), s));
      launches += 2;
    }
  }
  chk(cudaEventRecord(ws.ev1, s));
  std::vector<char> res_big(res_bytes <= kIoBytes ? 0 : res_bytes);
  char* const h_res = res_big.empty() ? ws.h_io : res_big.data();
  unsigned long long* const ctr = ws.h_stage;  // pinned
  chk(cudaMemcpyAsync(h_res, d_res, res_bytes, cudaMemcpyDeviceToHost, s));
  chk(cudaMemcpyAsync(ctr, sp.ctr, kCtrCount * 8, cudaMemcpyDeviceToHost, s));
  if (d_minp) chk(copy_out(ws, min_p_concat, d_minp, total_n * 4, s));
  chk(cudaStreamSynchronize(s));
  const uint64_t* psum = (const uint64_t*)h_res;
  const uint64_t* maxp = psum + count;
  const uint32_t* fails = (const uint32_t*)(maxp + count);
  float ms = 0;
  if (e == cudaSuccess) {
    cudaEventElapsedTime(&ms, ws.ev0, ws.ev1);
    if (o.mode == GB_WINDOWS_PERSISTENT) {
      cudaEventElapsedTime(&large_ms, ws.ek0, ws.ek1);
      cudaEventElapsedTime(&search_ms, ws.ek1, ws.ek2);
    }
  }
  if (e != cudaSuccess) return cuda_fail(ws, e, "windows");
  if (ctr[kCtrQueueOvf]) return fail(ws, GB_EOVERFLOW, "Phase-2 queue overflow: raise the halo");
  if (res) {
    for (size_t i = 0; i < count; ++i) {
      res[i].failures = fails[i];
      res[i].verified = w[i].count - fails[i];
      res[i].max_minp = maxp[i];
      res[i].minp_sum = psum[i];
    }
  }
  if (sum) {
    sum->total_n = total_n;
    sum->failures = ctr[kCtrFailures];
    sum->kernel_launches = launches;
    sum->device_ms = ms;
    sum->sieved_windows = nsw;
    sum->large_pairs = ctr[kCtrPairs];
    sum->large_ms = large_ms;
    sum->search_ms = search_ms;
  }
  return GB_OK;
}


// Windows that go n by n: every n of every window through the single-n kernel
// (minimal p over the resident table), then one per-window reduction.  Plain mode launches the single-n
// kernel window by window.
static gb_status windows_mr_impl(gb_ctx* c, Workspace& ws, Arena* arena, const gb_window* w,
                                 size_t count, const gb_windows_opts& o, uint64_t p_lim,
                                 gb_window_result* res, uint32_t* min_p_concat,
                                 gb_windows_summary* sum) {
  uint64_t total = 0;
  std::vector<uint64_t> off(count + 1, 0);
  for (size_t i = 0; i < count; ++i) off[i + 1] = off[i] + w[i].count;
  total = off[count];
  const uint64_t np = count_bound(c, p_lim);  // the kernel stops at p_lim itself
  gb_status st;
  ws.buf_used = 0;  // (as in windows_sieve_impl)
  Temps tmp(c, arena);
  void *d_w, *d_off, *d_n, *d_p, *d_q, *d_agg;
  if ((st = ws_buffer(c, ws, tmp, 0, count * sizeof(gb_window), &d_w)) != GB_OK ||
      (st = ws_buffer(c, ws, tmp, 1, (count + 1) * 8, &d_off)) != GB_OK ||
      (st = ws_buffer(c, ws, tmp, 2, total * 8, &d_n)) != GB_OK ||
      (st = ws_buffer(c, ws, tmp, 3, total * 8, &d_p)) != GB_OK ||
      (st = ws_buffer(c, ws, tmp, 4, total * 8, &d_q)) != GB_OK ||
      (st = ws_buffer(c, ws, tmp, 5, count * 32, &d_agg)) != GB_OK)
    return st;
  cudaStream_t s = o.stream ? (cudaStream_t)o.stream : c->stream;
  cudaError_t e = cudaSuccess;
  auto chk = [&](cudaError_t x) {
    if (e == cudaSuccess && x != cudaSuccess) e = x;
  };
  int launches = 0;
  chk(cudaEventRecord(ws.ev0, s));
  chk(cudaMemcpyAsync(d_w, w, count * sizeof(gb_window), cudaMemcpyHostToDevice, s));
  chk(cudaMemcpyAsync(d_off, off.data(), (count + 1) * 8, cudaMemcpyHostToDevice, s));
  chk(launch_win_expand((const gb_window*)d_w, (const uint64_t*)d_off, (uint32_t)count, (uint64_t*)d_n, s));
  ++launches;
  SingleArgs a{};
  a.primes = c->d_primes;
  a.nprimes = np;
  a.p_lim = p_lim;
  a.ctr = ws.ctr;
  const size_t parts = o.mode == GB_WINDOWS_PLAIN ? count : 1;
  for (size_t i = 0; i < parts && e == cudaSuccess; ++i) {
    const uint64_t b = parts == 1 ? 0 : off[i], n = parts == 1 ? total : w[i].count;
    a.n = (const uint64_t*)d_n + b;
    a.count = n;
    a.p_out = (uint64_t*)d_p + b;
    a.q_out = (uint64_t*)d_q + b;
    chk(cudaMemsetAsync(ws.ctr, 0, 4 * 8, s));
    chk(launch_single(a, c->sm_count, o.gpu_share_pct ? o.gpu_share_pct : 100, s));
    ++launches;
  }
  chk(launch_segment_reduce((const uint64_t*)d_p, (const uint64_t*)d_off, (uint32_t)count,
                            (unsigned long long*)d_agg, s));
  ++launches;
  chk(cudaEventRecord(ws.ev1, s));
  std::vector<unsigned long long> agg(count * 4);
  std::vector<uint64_t> pv(min_p_concat ? total : 0);
  chk(cudaMemcpyAsync(agg.data(), d_agg, count * 32, cudaMemcpyDeviceToHost, s));
  if (min_p_concat) chk(cudaMemcpyAsync(pv.data(), d_p, total * 8, cudaMemcpyDeviceToHost, s));
  chk(cudaStreamSynchronize(s));
  if (e != cudaSuccess) return cuda_fail(ws, e, "windows (n by n)");
  float ms = 0;
  cudaEventElapsedTime(&ms, ws.ev0, ws.ev1);
  uint64_t fails = 0;
  for (size_t i = 0; i < count; ++i) {
    if (res) {
      res[i].verified = agg[4 * i];
      res[i].failures = agg[4 * i + 1];
      res[i].max_minp = agg[4 * i + 2];
      res[i].minp_sum = agg[4 * i + 3];
    }
    fails += agg[4 * i + 1];
  }
  for (uint64_t j = 0; j < pv.size(); ++j) min_p_concat[j] = (uint32_t)pv[j];
  if (sum) {
    sum->total_n = total;
    sum->failures = fails;
    sum->kernel_launches = launches;
    sum->device_ms = ms;
  }
  return GB_OK;
}

// Splits the batch by path (per_n_windows): the windows taken n by n run through
// the single-n kernel, the others through the sieve pipeline.  Results do not
// depend on the split.
gb_status windows_impl(gb_ctx* c, Workspace& ws, Arena* arena, const gb_window* w, size_t count,
                       const gb_windows_opts* opts, gb_window_result* res, uint32_t* min_p_concat,
                       gb_windows_summary* sum) {
  gb_windows_opts o{};
  if (opts) o = *opts;
  if (!count || !w || o.on_device || o.mr_below == 1 ||
      (o.mode != GB_WINDOWS_PERSISTENT && o.mode != GB_WINDOWS_PLAIN))
    return windows_sieve_impl(c, ws, arena, w, count, opts, res, min_p_concat, sum);
  for (size_t i = 0; i < count; ++i) {
    const uint64_t last = w[i].start + 2 * (w[i].count - 1);
    if (w[i].start < 4 || (w[i].start & 1) || w[i].count == 0 || last < w[i].start)
      return windows_sieve_impl(c, ws, arena, w, count, opts, res, min_p_concat, sum);  // reports it
  }
  const uint64_t p_lim = o.phase2_limit ? o.phase2_limit : GB_PHASE2_LIMIT_DEFAULT;
  // (options that the pipeline refuses are refused for what it would take, and
  // its lockstep tries p = 3 whatever the bound)
  const bool few = opts_error(o) || p_lim < 3;
  const std::vector<char> narrow = per_n_windows(w, count, o, arena != nullptr, few);
  const size_t nn = std::count(narrow.begin(), narrow.end(), 1);
  if (nn == 0) return windows_sieve_impl(c, ws, arena, w, count, opts, res, min_p_concat, sum);
  if (p_lim > GB_P_SMALL_MAX) return fail(ws, GB_EINVAL, "phase2_limit must be <= 4e9");
  gb_status st = ensure_primes(c, ws, std::max<uint64_t>(p_lim, kWinChunkSieveBound));
  if (st != GB_OK) return st;
  // both parts in their own arrays, results put back in the caller's order
  std::vector<gb_window> wa, wb;
  std::vector<size_t> ia, ib;
  std::vector<uint64_t> out_off(count + 1, 0);
  for (size_t i = 0; i < count; ++i) {
    out_off[i + 1] = out_off[i] + w[i].count;
    (narrow[i] ? wa : wb).push_back(w[i]);
    (narrow[i] ? ia : ib).push_back(i);
  }
  std::vector<gb_window_result> ra(wa.size()), rb(wb.size());
  uint64_t na = 0, nb = 0;
  for (const gb_window& x : wa) na += x.count;
  for (const gb_window& x : wb) nb += x.count;
  std::vector<uint32_t> ma(min_p_concat ? na : 0), mb(min_p_concat ? nb : 0);
  gb_windows_summary sa{}, sb{};
  st = windows_mr_impl(c, ws, arena, wa.data(), wa.size(), o, p_lim, ra.data(),
                       min_p_concat ? ma.data() : nullptr, &sa);
  if (st == GB_ENOMEM && !o.mr_below && !few) {  // no room for their n (nothing launched yet): the pipeline alone
    ws.err.clear();
    return windows_sieve_impl(c, ws, arena, w, count, opts, res, min_p_concat, sum);
  }
  if (st != GB_OK) return st;
  if (!wb.empty() && (st = windows_sieve_impl(c, ws, arena, wb.data(), wb.size(), &o, rb.data(),
                                              min_p_concat ? mb.data() : nullptr, &sb)) != GB_OK)
    return st;
  uint64_t pa = 0, pb = 0;
  for (size_t k = 0; k < ia.size(); ++k) {
    if (res) res[ia[k]] = ra[k];
    if (min_p_concat) std::memcpy(min_p_concat + out_off[ia[k]], ma.data() + pa, wa[k].count * 4);
    pa += wa[k].count;
  }
  for (size_t k = 0; k < ib.size(); ++k) {
    if (res) res[ib[k]] = rb[k];
    if (min_p_concat) std::memcpy(min_p_concat + out_off[ib[k]], mb.data() + pb, wb[k].count * 4);
    pb += wb[k].count;
  }
  if (sum) {
    sum->total_n = sa.total_n + sb.total_n;
    sum->failures = sa.failures + sb.failures;
    sum->kernel_launches = sa.kernel_launches + sb.kernel_launches;
    sum->device_ms = sa.device_ms + sb.device_ms;
    sum->sieved_windows = sb.sieved_windows;
    sum->large_pairs = sb.large_pairs;
    sum->large_ms = sb.large_ms;
    sum->search_ms = sb.search_ms;
  }
  return GB_OK;
}

// Upper bound of the device bytes one window takes from a caller's arena in
// windows_impl: its share of the sieve path's buffers (descriptor, record,
// offsets, results, class masks) or, when it is narrow enough to go n by n, of
// that path's (its n, p, q and a reduction record), whichever is more; arena
// alignment included.  Used by serving to admit batches by memory.
uint64_t windows_request_bytes(const gb_window& w, const gb_windows_opts& o) {
  const uint64_t H = o.halo ? o.halo : kWinHalo;
  const uint64_t fixed = sizeof(WinDesc6) + sizeof(WinLarge) + 88 + 4 + 16 + 16 + 4 * 256;
  const uint64_t lwords = (w.count / 3 + H / 6 + 96) / 32 + 16;
  const bool per_n = o.mr_below ? w.count < o.mr_below && o.mr_below != 1 : is_narrow(w);
  return fixed + std::max(2 * lwords * 4, per_n ? w.count * 24 + 64 + 4 * 256 : 0);
}

// Autotuner of the windows pipeline: the persistent mode on a sample of the
// batch (every k-th window, at most 512) for each candidate, after one
// warm-up call; the fastest device time wins.  Cached per batch class.
gb_status autotune_windows_impl(gb_ctx* c, Workspace& ws, const gb_window* w, size_t count,
                                const gb_windows_opts* base, gb_windows_opts* tuned,
                                gb_windows_tune* res) {
  if (!tuned || (count && !w)) return fail(ws, GB_EINVAL, "null argument");
  gb_windows_opts o{};
  if (base) o = *base;
  *tuned = o;
  gb_windows_tune r{};
  if (count == 0) {
    if (res) *res = r;
    return GB_OK;
  }
  uint64_t top = 0;
  for (size_t i = 0; i < count; ++i) top = std::max<uint64_t>(top, w[i].start + 2 * (w[i].count - 1));
  uint64_t tb = 0, cb = 0;
  for (uint64_t x = top; x; x >>= 1) ++tb;
  for (uint64_t x = count; x; x >>= 1) ++cb;
  const std::vector<uint64_t> key{tb, cb, o.phase2_limit};
  auto it = c->tuned_windows.find(key);
  if (it != c->tuned_windows.end()) {
    r = it->second;
    r.candidates = 0;
    r.cached = 1;
  } else {
    const size_t step = (count + 511) / 512;
    std::vector<gb_window> smp;
    for (size_t i = 0; i < count; i += step) smp.push_back(w[i]);
    std::vector<gb_window_result> wr(smp.size());
    gb_windows_opts t = o;
    t.mode = GB_WINDOWS_PERSISTENT;
    t.on_device = 0;
    gb_windows_summary sum{};
    gb_status st = windows_impl(c, ws, nullptr, smp.data(), smp.size(), &t, wr.data(), nullptr, &sum);
    if (st != GB_OK) return st;  // warm-up (tables)
    uint64_t n = 0;
    for (const gb_window& x : smp) n += x.count;
    double best = -1;
    for (uint32_t div : {30u, 20u, 45u})
      for (uint32_t chunk : {1u << 20, 1u << 19})
        for (uint32_t large : {64u, 16u})
          for (uint32_t threads : {512u, 256u}) {
            t.mr_divisor = div;
            t.chunk_evens = chunk;
            t.large_ctas_per_sm = large;
            t.block_threads = threads;
            if ((st = windows_impl(c, ws, nullptr, smp.data(), smp.size(), &t, wr.data(), nullptr,
                                   &sum)) != GB_OK)
              return st;
            ++r.candidates;
            const double rate = sum.device_ms > 0 ? n / (sum.device_ms / 1e3) : 0;
            if (rate > best) {
              best = rate;
              r.mr_divisor = div;
              r.chunk_evens = chunk;
              r.large_ctas_per_sm = large;
              r.block_threads = threads;
            }
          }
    r.even_n_per_s = best;
    r.sample_windows = (uint32_t)smp.size();
    c->tuned_windows[key] = r;
  }
  tuned->mr_divisor = r.mr_divisor;
  tuned->chunk_evens = r.chunk_evens;
  tuned->large_ctas_per_sm = r.large_ctas_per_sm;
  tuned->block_threads = r.block_threads;
  if (res) *res = r;
  return GB_OK;
}

}  // namespace gb
