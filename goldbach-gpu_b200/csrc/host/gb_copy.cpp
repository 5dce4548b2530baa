// gb_copy.cpp -- device -> host copies of a call's large outputs.
#include <algorithm>
#include <atomic>
#include <chrono>
#include <condition_variable>
#include <cstring>
#include <mutex>
#include <thread>

#include "gb_ctx.h"

namespace gb {

// A pageable copy of the runtime moves about 6.5 GB/s; the ring's slots come in at
// the link's rate and four threads empty them.  Starting and joining the threads
// takes up to half a millisecond, so smaller copies stay with the runtime.
// Range calls with per-n output into a fresh numpy array, median us, runtime / ring: 4 MB 421
// / 588, 8 MB 714 / 790, 11 MB 916 / 885, 32 MB 7630 / 3420; into one used before:
// 11 MB 776 / 707, 16 MB 1075 / 1057, 64 MB 4030 / 3156.
constexpr size_t kRingSlot = 1u << 20, kRingLeast = 10u << 20;
constexpr int kRingSlots = 4, kRingThreads = 4;

// The ring's memory and events, all of them or none.
static bool ring_init(Workspace& w) {
  void* ring = nullptr;
  cudaEvent_t ev[kRingSlots] = {};
  bool ok = cudaMallocHost(&ring, kRingSlot * kRingSlots) == cudaSuccess;
  for (cudaEvent_t& e : ev) ok = ok && cudaEventCreateWithFlags(&e, cudaEventDisableTiming) == cudaSuccess;
  if (!ok) {
    for (cudaEvent_t e : ev)
      if (e) cudaEventDestroy(e);
    if (ring) cudaFreeHost(ring);
    cudaGetLastError();
    return false;
  }
  w.h_ring = (char*)ring;
  std::copy(ev, ev + kRingSlots, w.ring_ev);
  return true;
}

cudaError_t copy_out(Workspace& w, void* dst, const void* src, size_t bytes, cudaStream_t s) {
  cudaPointerAttributes at{};
  if (bytes < kRingLeast ||
      (cudaPointerGetAttributes(&at, dst) == cudaSuccess && at.type != cudaMemoryTypeUnregistered))
    return cudaMemcpyAsync(dst, src, bytes, cudaMemcpyDeviceToHost, s);
  cudaGetLastError();
  if (!w.h_ring && !ring_init(w)) return cudaMemcpyAsync(dst, src, bytes, cudaMemcpyDeviceToHost, s);
  const size_t slots = (bytes + kRingSlot - 1) / kRingSlot;
  auto len = [&](size_t i) { return std::min(kRingSlot, bytes - i * kRingSlot); };
  auto fill = [&](size_t i) {
    const int r = (int)(i % kRingSlots);
    cudaError_t x = cudaMemcpyAsync(w.h_ring + r * kRingSlot, (const char*)src + i * kRingSlot, len(i),
                                    cudaMemcpyDeviceToHost, s);
    return x == cudaSuccess ? cudaEventRecord(w.ring_ev[r], s) : x;
  };
  // ready: slots that have arrived; taken: the next quarter of a slot to empty;
  // left: quarters of each ring slot not yet emptied
  std::atomic<size_t> ready{0}, taken{0};
  std::atomic<int> left[kRingSlots];
  constexpr size_t kParts = 4;
  for (auto& l : left) l.store(0);
  auto empty_one = [&]() -> bool {  // whether there was a part to take
    size_t t = taken.load(std::memory_order_relaxed);
    do {
      if (t >= ready.load(std::memory_order_acquire) * kParts) return false;
    } while (!taken.compare_exchange_weak(t, t + 1));
    const size_t i = t / kParts, part = len(i) / kParts, o = (t % kParts) * part;
    const size_t n = t % kParts == kParts - 1 ? len(i) - o : part;
    std::memcpy((char*)dst + i * kRingSlot + o, w.h_ring + (i % kRingSlots) * kRingSlot + o, n);
    left[i % kRingSlots].fetch_sub(1, std::memory_order_release);
    return true;
  };
  // The kernels that make the bytes may run for long: until they are behind, this
  // thread waits in the runtime, and the helpers go to sleep after a millisecond.
  // (Asleep from the start they wake 45 us late: 61 windows with per-n output
  // 1.16 ms instead of 1.11.)
  std::mutex mu;
  std::condition_variable cv;
  std::atomic<bool> behind{false};
  std::atomic<bool> stop{false};
  std::thread helpers[kRingThreads - 1];
  int nh = 0;
  try {
    for (; nh < kRingThreads - 1; ++nh)
      helpers[nh] = std::thread([&] {
        const auto until = std::chrono::steady_clock::now() + std::chrono::milliseconds(1);
        while (!behind.load(std::memory_order_acquire) && std::chrono::steady_clock::now() < until)
          std::this_thread::yield();
        if (!behind.load(std::memory_order_acquire)) {
          std::unique_lock<std::mutex> lk(mu);
          cv.wait(lk, [&] { return behind.load(); });
        }
        while (!stop.load(std::memory_order_acquire))
          if (!empty_one()) std::this_thread::yield();
      });
  } catch (...) {  // no more threads: fewer helpers
  }
  // (the last ring slot's event stands in front of the copies until then)
  const size_t last = kRingSlots - 1;
  cudaError_t e = cudaEventRecord(w.ring_ev[last], s);
  for (size_t i = 0; i < slots && i < last && e == cudaSuccess; ++i) e = fill(i);
  if (e == cudaSuccess) e = cudaEventSynchronize(w.ring_ev[last]);
  {
    std::lock_guard<std::mutex> lk(mu);
    behind.store(true, std::memory_order_release);
  }
  cv.notify_all();
  if (slots > last && e == cudaSuccess) e = fill(last);
  for (size_t i = 0; i < slots && e == cudaSuccess; ++i) {
    const int r = (int)(i % kRingSlots);
    while (e == cudaSuccess) {  // slot i's arrival, emptying earlier ones meanwhile
      const cudaError_t q = cudaEventQuery(w.ring_ev[r]);
      if (q == cudaSuccess) break;
      if (q != cudaErrorNotReady) e = q;
      empty_one();
    }
    cudaGetLastError();
    if (e != cudaSuccess) break;
    left[r].store((int)kParts, std::memory_order_relaxed);
    ready.store(i + 1, std::memory_order_release);
    if (i + 1 >= (size_t)kRingSlots && i + 1 < slots) {  // slot i + 1 goes where slot i + 1 - kRingSlots was
      while (left[(i + 1) % kRingSlots].load(std::memory_order_acquire) != 0) empty_one();
      e = fill(i + 1);
    }
  }
  while (e == cudaSuccess && empty_one()) {
  }
  for (auto& l : left)
    while (e == cudaSuccess && l.load(std::memory_order_acquire) != 0) std::this_thread::yield();
  stop.store(true, std::memory_order_release);
  for (int h = 0; h < nh; ++h) helpers[h].join();
  return e;
}

}  // namespace gb
