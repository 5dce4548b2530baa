"""copy_out (goldbach-gpu_b200/csrc/host/gb_copy.cpp) on the host, over a small
stand-in for the CUDA runtime: one stream whose work a thread runs in order,
behind a kernel of a given length, and calls that can be made to fail.  The
pinned ring's copies arrive whole, small ones do without it, a ring that could
not be set up leaves nothing behind that a later copy trips over, and the threads
that empty the ring sleep while the kernel in front of the copy runs."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.abspath(os.path.join(os.path.dirname(__file__), ".."))
CSRC = os.path.join(ROOT, "goldbach-gpu_b200", "csrc")
CUDA = os.environ.get("CUDA", "/usr/local/cuda")

_HARNESS = r"""
#include <chrono>
#include <condition_variable>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <ctime>
#include <deque>
#include <functional>
#include <mutex>
#include <thread>

#include "host/gb_ctx.h"

// -- the stand-in ---------------------------------------------------------------
struct Ev { bool done = false; };
static std::mutex mu;
static std::condition_variable cv;
static std::deque<std::function<void()>> stream;
static bool idle = true;
static int fail_event = -1;           // the event creation that fails, counted down
static bool fail_host = false;
static int events = 0, pinned = 0;    // alive

static void worker() {
  for (;;) {
    std::unique_lock<std::mutex> lk(mu);
    cv.wait(lk, [] { return !stream.empty(); });
    auto f = stream.front();
    idle = false;
    lk.unlock();
    f();
    lk.lock();
    stream.pop_front();
    idle = stream.empty();
    cv.notify_all();
  }
}
static void push(std::function<void()> f) {
  std::lock_guard<std::mutex> lk(mu);
  stream.push_back(std::move(f));
  idle = false;
  cv.notify_all();
}
static void drain() {
  std::unique_lock<std::mutex> lk(mu);
  cv.wait(lk, [] { return idle; });
}

extern "C" {
cudaError_t cudaPointerGetAttributes(cudaPointerAttributes* a, const void*) {
  a->type = cudaMemoryTypeUnregistered;
  return cudaSuccess;
}
cudaError_t cudaGetLastError(void) { return cudaSuccess; }
cudaError_t cudaMallocHost(void** p, size_t n) {
  if (fail_host) return cudaErrorMemoryAllocation;
  *p = malloc(n);
  ++pinned;
  return cudaSuccess;
}
cudaError_t cudaHostAlloc(void** p, size_t n, unsigned) { return cudaMallocHost(p, n); }
cudaError_t cudaFreeHost(void* p) {
  free(p);
  --pinned;
  return cudaSuccess;
}
cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, unsigned) {
  if (fail_event >= 0 && fail_event-- == 0) return cudaErrorMemoryAllocation;
  *e = (cudaEvent_t) new Ev;
  ++events;
  return cudaSuccess;
}
cudaError_t cudaEventDestroy(cudaEvent_t e) {
  delete (Ev*)e;
  --events;
  return cudaSuccess;
}
cudaError_t cudaEventRecord(cudaEvent_t e, cudaStream_t) {
  if (!e) return cudaErrorInvalidResourceHandle;
  {
    std::lock_guard<std::mutex> lk(mu);
    ((Ev*)e)->done = false;
  }
  push([e] {
    std::lock_guard<std::mutex> lk(mu);
    ((Ev*)e)->done = true;
  });
  return cudaSuccess;
}
cudaError_t cudaEventQuery(cudaEvent_t e) {
  std::lock_guard<std::mutex> lk(mu);
  return ((Ev*)e)->done ? cudaSuccess : cudaErrorNotReady;
}
cudaError_t cudaEventSynchronize(cudaEvent_t e) {
  std::unique_lock<std::mutex> lk(mu);
  cv.wait(lk, [e] { return ((Ev*)e)->done; });
  return cudaSuccess;
}
cudaError_t cudaMemcpyAsync(void* d, const void* s, size_t n, cudaMemcpyKind, cudaStream_t) {
  push([=] { std::memcpy(d, s, n); });
  return cudaSuccess;
}
}
template <class T>
static bool same(const T& a, const T& b) { return !std::memcmp(a.data(), b.data(), a.size()); }

static std::vector<char> pattern(size_t n, unsigned seed) {
  std::vector<char> v(n);
  for (char& c : v) c = (char)((seed = seed * 1664525u + 1013904223u) >> 24);
  return v;
}
static int fails = 0;
static void check(bool ok, const char* what) {
  if (!ok) ++fails, std::printf("FAIL %s\n", what);
}
static bool copies(gb::Workspace& w, size_t n, unsigned seed) {
  const std::vector<char> src = pattern(n, seed);
  std::vector<char> dst(n);
  const cudaError_t e = gb::copy_out(w, dst.data(), src.data(), n, nullptr);
  drain();
  return e == cudaSuccess && same(src, dst);
}

int main(int argc, char** argv) {
  std::thread(worker).detach();
  const std::string mode = argc > 1 ? argv[1] : "";
  if (mode == "sizes") {
    gb::Workspace w;
    const size_t m = 1 << 20;
    unsigned seed = 0;
    for (size_t n : {size_t(1), m, 10 * m - 1}) {
      check(copies(w, n, ++seed), "copy");
      check(pinned == 0 && events == 0, "a small copy sets up no ring");
    }
    for (size_t n : {10 * m, 10 * m + 1, 12 * m - 1, 12 * m + 3, 37 * m + 12345})
      check(copies(w, n, ++seed), "copy");
    check(pinned == 1, "the ring");
  } else if (mode == "setup") {
    for (int k = 0; k < 5; ++k) {  // the k-th event, or (4) the memory, cannot be had
      gb::Workspace w;
      const int ev = events, pin = pinned;
      fail_event = k < 4 ? k : -1;
      fail_host = k == 4;
      check(copies(w, 11 << 20, k), "copy without a ring");
      check(events == ev && pinned == pin, "nothing kept");
      fail_event = -1;
      fail_host = false;
      check(copies(w, 11 << 20, 10 + k), "the next copy");
      check(copies(w, 13 << 20, 20 + k), "and the one after");
      check(events == ev + 4 && pinned == pin + 1, "the ring");
    }
  }
  if (mode == "kernel") {  // a kernel of 0.4 s in front: the host waits, it does not work
    gb::Workspace w;
    check(copies(w, 11 << 20, 1), "the first copy");
    push([] { std::this_thread::sleep_for(std::chrono::milliseconds(400)); });
    const std::clock_t c0 = std::clock();  // of all threads
    check(copies(w, 11 << 20, 2), "the copy behind it");
    check((double)(std::clock() - c0) / CLOCKS_PER_SEC < 0.2, "processor time");
  }
  std::printf(fails ? "failed\n" : "ok\n");
  std::fflush(stdout);
  std::_Exit(fails ? 1 : 0);  // (the stream's thread waits for work)
}
"""


@pytest.fixture(scope="module")
def harness(tmp_path_factory):
    if shutil.which("g++") is None or not os.path.isdir(os.path.join(CUDA, "include")):
        pytest.skip("needs g++ and the CUDA headers")
    d = tmp_path_factory.mktemp("copy_out")
    src, exe = d / "harness.cpp", d / "harness"
    src.write_text(_HARNESS)
    subprocess.run(["g++", "-std=c++17", "-O2", "-I", CSRC, "-I", os.path.join(ROOT, "include"), "-I",
                    os.path.join(CUDA, "include"), "-o", str(exe), str(src), os.path.join(CSRC, "host", "gb_copy.cpp"),
                    "-lpthread"], check=True, capture_output=True, text=True, timeout=120)
    return str(exe)


@pytest.mark.parametrize("mode", ["sizes", "setup", "kernel"])
def test_copy_out(harness, mode):
    r = subprocess.run([harness, mode], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0 and r.stdout.strip().endswith("ok"), r.stdout[-2000:]
