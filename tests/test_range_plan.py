"""How a range is cut (goldbach-gpu_b200/csrc/host/range_plan.h), compiled on the
host: chunk widths are multiples of 512 within their bounds and no wider than
the longest piece, whatever the number of pieces."""
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

int main() {
  widths();
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
