"""How a range is cut (goldbach-gpu_b200/csrc/host/range_plan.h), compiled on the
host: chunk widths are multiples of 512 within their bounds and no wider than
the longest piece, whatever the number of pieces, and the large-prime masks are
taken where they were measured to pay."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.abspath(os.path.join(os.path.dirname(__file__), ".."))
HOST = os.path.join(ROOT, "goldbach-gpu_b200", "csrc", "host")

_HARNESS = r"""
#include <cstdio>
#include <random>
#include "range_plan.h"

static int fails = 0;
static void check(bool ok, const char* what, unsigned long long a, unsigned long long b, unsigned long long c) {
  if (!ok && fails++ < 20) std::printf("FAIL %s: %llu %llu %llu\n", what, a, b, c);
}

static void widths() {
  std::mt19937_64 rng(5);
  for (int i = 0; i < 200000; ++i) {
    const int sm = i % 3 ? 148 : 1 + (int)(rng() % 200);
    const uint64_t pieces = rng() % 4 ? rng() >> (44 + rng() % 20) : 0, len = 1 + (rng() >> (20 + rng() % 43));
    const uint64_t tail = rng() % 3 ? rng() % len : 0;
    const uint32_t least = rng() % 2 ? 8192 : 65536, most = rng() % 2 ? 1u << 20 : 65536;
    const double fixed = 1e5 + (double)(rng() % 30000000);
    const uint32_t ne = gb::balanced_chunk(pieces, len, tail, fixed, sm, least, most);
    check(ne >= least && ne <= most && ne % 512 == 0, "width", ne, least, most);
    const uint64_t longest = pieces ? len : tail;  // tail < len
    check(ne == least || ne < longest + 512, "no wider than a piece", ne, pieces, longest);
  }
}

// us per call of the chunks alone and of the masks (B200, 148 SMs): the rule takes
// the faster one, or one within a tenth of it
static void masks() {
  struct Case { double top, count, seg; int shards; double alone, masked; };
  const Case cases[] = {
      {9e9, 1e5, 1e7, 1, 93, 114},      {9e9, 1e7, 1e3, 1, 973, 1408},    {9e9, 1e7, 1e3, 2, 532, 3092},
      {9e9, 1e7, 3e3, 2, 247, 966},     {9e9, 1e7, 1e7, 1, 111, 150},     {1e11, 1e6, 1e7, 1, 115, 117},
      {1e11, 1e7, 3e3, 2, 330, 971},    {1e12, 1e5, 1e7, 1, 138, 118},    {1e12, 1e6, 1e3, 1, 332, 231},
      {1e12, 1e7, 1e3, 1, 2379, 1496},  {1e12, 1e7, 1e3, 2, 1241, 3059},  {1e12, 1e7, 3e3, 2, 508, 980},
      {1e12, 1e7, 1e4, 2, 233, 319},    {1e12, 1e7, 1e7, 1, 144, 152},    {4e12, 1e7, 1e7, 1, 185, 157},
      {4e12, 3e7, 1e7, 1, 207, 208},    {1e13, 1e6, 1e3, 1, 627, 231},    {1e13, 1e7, 1e3, 2, 2604, 3346},
      {1e13, 1e7, 3e4, 2, 243, 212},    {1e13, 1e7, 1e7, 1, 220, 165},    {1e13, 1e8, 1e7, 1, 319, 500},
      {5e13, 1e9, 1e7, 1, 2038, 1906},  {1e14, 1e7, 1e3, 2, 6536, 4118},  {1e14, 1e8, 1e7, 1, 527, 318},
  };
  for (const Case& c : cases) {
    const uint64_t root = (uint64_t)std::sqrt(c.top), segs = (uint64_t)std::ceil(c.count / c.seg);
    const uint64_t mine = (segs + c.shards - 1) / c.shards;
    const bool m = gb::range_masked_pays(148, (uint64_t)(c.top - 2 * c.count), (uint64_t)(c.count / c.shards), root, mine,
                                         c.shards > 1 ? mine : 1, 1u << 20, segs);
    check((m ? c.masked : c.alone) <= 1.1 * std::min(c.masked, c.alone), "masks", (uint64_t)c.top, (uint64_t)c.count,
          (uint64_t)c.seg);
  }
  // below every sieving prime, and with more segments than the descriptors are meant for
  check(!gb::range_masked_pays(148, 1u << 30, 1000, 1u << 20, 1, 1, 8192, 1), "low", 0, 0, 0);
  check(!gb::range_masked_pays(148, 1ull << 60, 1ull << 40, 1u << 30, (1u << 20) + 1, 1, 8192, (1u << 20) + 1), "pieces", 0, 0, 0);
}

// a segment is cut into runs of 2^28 n, each with descriptors of its own
static void descriptors() {
  check(gb::range_masked_pays(148, 1ull << 60, 1ull << 47, 1u << 30, 100, 1, 8192, 100), "2^19 runs", 0, 0, 0);
  for (uint64_t n : {1ull << 49, 1ull << 55, 1ull << 62})
    check(!gb::range_masked_pays(148, 1ull << 40, n, 0xffffffffu, 1, 1, 8192, 1), "one segment's runs", n, 0, 0);
}

// a piece carries its segment's index in the whole range in 32 bits
static void indexes() {
  for (int k : {-1, 0, 1})
    check(gb::range_masked_pays(148, 1ull << 60, 1u << 20, 1u << 30, 1000, 1000, 8192, (1ull << 32) + k) == (k < 0),
          "segments", k + 1, 0, 0);
}

int main() {
  widths();
  masks();
  descriptors();
  indexes();
  std::printf(fails ? "failed\n" : "ok\n");
  return fails ? 1 : 0;
}
"""


@pytest.mark.skipif(shutil.which("g++") is None, reason="needs g++")
def test_range_plan(tmp_path):
    src, exe = tmp_path / "plan.cpp", tmp_path / "plan"
    src.write_text(_HARNESS)
    subprocess.run(["g++", "-std=c++17", "-O2", "-Wall", "-Werror", "-I", HOST, "-o", str(exe), str(src)],
                   check=True, capture_output=True, text=True, timeout=120)
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0 and r.stdout.strip().endswith("ok"), r.stdout[-2000:]
